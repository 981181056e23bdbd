"""The workloads that this framework's speed is judged by, through its public entry points.

Each case is work that a flow code has the pressure solver do: a solve by
each of the FFVILS methods (RBGS, CG, BiCGSTAB) and by the mixed-precision
form, from the smallest grid (16 leaf blocks) to the 4692-block level-5
sphere grid; a batch of independent problems; a whole fractional time step
and a solve whose fields live on the host, transfers included; and a loop of
single calls.  Grids are octrees of 16^3-cell leaf blocks refined around a
sphere; u* = (1, 0, 0) + noise and the cut cells of the sphere go through the
cut-cell assembly, as a flow code's do.

Solves are cut off at a stated number of iterations ('count'), below what
1e-8 takes, so that a case's work is known; they poll for convergence as a
solve to 1e-8 does (RBGS cases that state eps = 0 do not).  BiCGSTAB's iterates
amplify rounding about tenfold every few iterations, so its cases stop while
they still agree with a 64-bit restatement that rounds in another order.

exact() restates the same path in plain torch, in 64 bits, on [block][k][j][i]
arrays: octree, exchange, assembly, solvers, projection.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "ffv-hc_b200"))
import ffvgpu  # noqa: E402

VC = 2                    # guide width of host arrays (the reference's default)
W = 16 + 2 * VC
ORIGIN = (-4.0, -4.0, -4.0)
RHOF, DT, SIGMA = 1.0, 0.002, 0.01
A_FIELDS = ("AP", "AW", "AE", "AS", "AN", "AB", "AT")
U_FIELDS = ("UX", "UY", "UZ")


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def _grid(level, root=(4, 2, 2), center=(0.0, 0.0, 0.0), radius=0.5):
    return dict(level=level, gx=root[0], gy=root[1], gz=root[2], cx=center[0], cy=center[1],
                cz=center[2], radius=radius)


def listed():
    return [
        # a caller's own loop of single calls on the smallest grid (16 blocks): latency
        dict(name="calls_16", kind="calls", omega=1.2, count=4, **_grid(0)),
        # a coarse grid solved by RBGS: launch latency counts (72 blocks)
        dict(name="rbgs_72", kind="rbgs", omega=1.1, count=100, eps=1e-8, **_grid(1)),
        # an ordinary RBGS solve on a grid whose block count divides by nothing handy
        dict(name="rbgs_odd", kind="rbgs", omega=1.0, count=200, eps=1e-8,
             **_grid(3, (3, 3, 1), (1.3, 0.9, -2.1), 0.6)),
        # the benchmark's headline solve: 4692 blocks, 200 sweeps, a residual after each
        dict(name="rbgs_level5", kind="rbgs", omega=1.5, count=200, eps=0.0, **_grid(5)),
        # the reference's default solver on a small grid (128 blocks)
        dict(name="bicgstab_128", kind="bicgstab", omega=1.0, pre=2, count=24, eps=1e-8, drop=0.0,
             **_grid(2)),
        # and on the at-scale grid, with the restarts that grid needs
        dict(name="bicgstab_level5", kind="bicgstab", omega=1.0, pre=2, count=24, eps=1e-8,
             drop=1e-3, **_grid(5)),
        # CG, PreCount 3, on the 548-block grid
        dict(name="cg_548", kind="cg", omega=1.0, pre=3, count=40, eps=1e-8, **_grid(3)),
        # the mixed form with its FP64-data option, mid-sized grid
        dict(name="mixed_fp64data", kind="mixed", omega=1.5, sweeps=8, per=4, count=32, eps=1e-8,
             fp64=True, **_grid(3, (3, 2, 2), (0.7, -1.2, 0.4), 0.8)),
        # the mixed form at scale
        dict(name="mixed_level5", kind="mixed", omega=1.5, sweeps=8, per=4, count=40, eps=1e-8,
             fp64=False, **_grid(5)),
        # independent problems of mixed sizes solved together
        dict(name="batch_16", kind="batch", omega=1.5, sweeps=8, per=4, count=24, eps=1e-8,
             instances=16, layout=3, **_grid(4)),
        # one fractional step of a host flow code: u* and p up, UpdateP + UpdateU, u and p down
        dict(name="step_1164", kind="step", omega=1.0, pre=2, count=20, eps=1e-8, drop=1e-3,
             **_grid(4)),
        # a drop-in solve whose A, b and x live on the host: all up, RBGS, x down
        dict(name="host_solve_1164", kind="host", omega=1.0, count=20, eps=1e-8, **_grid(4)),
    ]


MAX_CELL_SWEEPS = 4692 * 200  # blocks x sweeps of the largest listed case
# blocks x iterations that cost as much, per kind (an iteration's passes against a sweep's)
COST = {"calls": 1, "rbgs": 1, "bicgstab": 5, "cg": 4, "mixed": 6, "batch": 6}


def _draw_grid(rng, top):
    level = rng.randint(0, top)
    root = (rng.randint(2, 4), rng.randint(1, 3), rng.randint(1, 3))
    ext = [4.0 * r for r in root]
    center = [round(ORIGIN[a] + ext[a] * rng.uniform(0.25, 0.75), 3) for a in range(3)]
    return _grid(level, root, center, round(rng.uniform(0.25, 0.9), 3))


def draw(rng):
    while True:
        kind = rng.choice(("calls", "rbgs", "rbgs", "bicgstab", "bicgstab", "cg", "mixed",
                           "mixed", "batch", "step", "host"))
        c = dict(kind=kind, **_draw_grid(rng, 4 if kind in ("step", "host", "batch") else 5))
        log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
        if kind == "calls":
            c.update(omega=round(rng.uniform(0.8, 1.2), 2), count=rng.randint(1, 8))
        elif kind == "rbgs":
            c.update(omega=round(rng.uniform(0.8, 1.2), 2), count=log(20, 200),
                     eps=rng.choice((0.0, 1e-8)))
        elif kind == "bicgstab":
            c.update(omega=1.0, pre=rng.randint(1, 3), count=log(5, 24), eps=1e-8,
                     drop=rng.choice((0.0, 1e-3)))
        elif kind == "cg":
            c.update(omega=1.0, pre=rng.randint(1, 3), count=log(10, 40), eps=1e-8)
        elif kind in ("mixed", "batch"):
            per = rng.choice((2, 4, 8))
            c.update(omega=rng.choice((1.2, 1.5)), sweeps=per * rng.randint(1, 2), per=per,
                     count=log(8, 40), eps=1e-8)
            if kind == "mixed":
                c.update(fp64=rng.random() < 0.4)
            else:
                c.update(instances=rng.randint(2, 16), layout=rng.randint(0, 10 ** 6))
        else:
            c.update(omega=1.0, count=log(5, 20), eps=1e-8)
            if kind == "step":
                c.update(pre=rng.randint(1, 3), drop=1e-3)
        nb = _total_blocks(c)
        if kind in ("step", "host"):
            if nb <= 1164:
                return c
        elif COST[kind] * nb * c["count"] <= MAX_CELL_SWEEPS * 1.2 and nb <= 9000:
            return c


# ---------------------------------------------------------------------------
# What a user's program has in hand, and the passes
# ---------------------------------------------------------------------------
def _sphere(case):
    return dict(root_grid=(case["gx"], case["gy"], case["gz"]),
                center=(case["cx"], case["cy"], case["cz"]), radius=case["radius"])


def _batch_problems(case, seed):
    """The batch's independent problems: grids (fixed by 'layout') of levels up to the case's."""
    rng = np.random.RandomState(case["layout"])
    out = []
    for n in range(case["instances"]):
        g = _grid(int(rng.randint(min(1, case["level"]), case["level"] + 1)), (4, 2, 2),
                  [float(np.round(rng.uniform(-1.0, 1.0), 3)) for _ in range(3)],
                  float(np.round(rng.uniform(0.25, 0.7), 3)))
        out.append((g, 1000 * seed + n))
    return out


def _total_blocks(case):
    if case["kind"] == "batch":
        return sum(len(_leaves(_key(g))[0]) for g, _ in _batch_problems(case, 0))
    return len(_leaves(_key(case))[0])


_PINNED = {}


def _pinned(dtype, n):
    """A reused pinned host buffer: uploads end before it is filled again."""
    b = _PINNED.get(dtype)
    if b is None or b.numel() < n:
        b = _PINNED[dtype] = torch.empty(n, dtype=dtype, pin_memory=True)
    return b[:n]


def _padded(t):
    """[nb][16][16][16] -> the reference's host layout, guide cells 0."""
    return torch.nn.functional.pad(t, (VC,) * 6)


def _upload(pool, field, t):
    t = _padded(t)
    h = _pinned(t.dtype, t.numel())
    h.copy_(t.reshape(-1))
    torch.cuda.synchronize()
    pool.upload_ptr(field, h.data_ptr(), VC)


def _assembled_pool(case, seed):
    """A pool with A and b assembled from u* and the sphere's cut cells, x = 0."""
    g = ffvgpu.SphereGrid(case["level"], **_sphere(case))
    pool = ffvgpu.Pool(g.desc())
    inp = _inputs(g.level, g.index, case, seed)
    for name, t in inp.items():
        _upload(pool, name, t)
    for u in U_FIELDS:
        pool.exchange(u, ffvgpu.U_BC_TYPE, ffvgpu.U_BC_VALUE[u])
    pool.assemble_p(RHOF, DT)
    pool.fold_bc()
    pool.fill("X", 0.0)
    return g, pool


def _host(nb):
    return torch.empty((nb, W, W, W), dtype=torch.float64, pin_memory=True)


class _PoolArray(ffvgpu._DeviceArray):
    """A pool's device array that keeps the pool alive as long as a tensor views it."""

    def __init__(self, owner, ptr, blocks):
        super().__init__(ptr, (blocks, 4096))
        self.owner = owner


def _iterate(owner, blocks):
    """torch view of the pressure (pool_iterate, with the pool's lifetime tied to the tensor)."""
    ptr = ctypes.c_void_p()
    st = ffvgpu.lib().ffvgpu_pool_field_device(owner._h, ffvgpu.FIELD["X"], ctypes.byref(ptr))
    assert st == ffvgpu.OK, st
    return torch.as_tensor(_PoolArray(owner, ptr.value, blocks), device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        probs = _batch_problems(case, seed)
        n = _total_blocks(case)
        batch = ffvgpu.Batch(n, len(probs))
        ids = [batch.admit_sphere(ffvgpu.sphere_problem(g["level"], seed=s, sigma=SIGMA, dt=DT,
                                                        rhof=RHOF, **_sphere(g)))
               for g, s in probs]
        return dict(case=case, batch=batch, ids=ids, n=n)
    g, pool = _assembled_pool(case, seed)
    st = dict(case=case, pool=pool, nb=g.nb)
    if kind == "step":
        # the flow code's own arrays: u* and the last pressure, and where results go
        f = _step_fields(g.level, g.index, case, seed)
        st["up"] = {k: _host(g.nb).copy_(v) for k, v in f.items()}
        st["down"] = {k: _host(g.nb) for k in f}
    elif kind == "host":
        st["up"] = {k: _host(g.nb) for k in A_FIELDS + ("B",)}
        for k, h in st["up"].items():
            pool.download_ptr(k, h.data_ptr(), VC)
        st["up"]["X"] = _host(g.nb).zero_()
        st["x"] = _host(g.nb)
    return st


def run(st):
    c = st["case"]
    kind = c["kind"]
    if kind == "batch":
        b = st["batch"]
        for i in st["ids"]:
            b.fill(i, "X", 0.0)
        r = b.solve_mixed(omega=c["omega"], sweeps=c["sweeps"], sweeps_per_exchange=c["per"],
                          count_max=c["count"], epsilon=c["eps"])
        return dict(x=_iterate(b, st["n"]), count=r["count"], residual=r["residual"])
    p = st["pool"]
    if kind == "step":
        for k, h in st["up"].items():
            p.upload_ptr(k, h.data_ptr(), VC)
        r = p.update_p(omega=c["omega"], pre_count=c["pre"], count_max=c["count"],
                       epsilon=c["eps"], restart_drop=c["drop"], rhof=RHOF, dt=DT)
        p.update_u(RHOF, DT)
        for k, h in st["down"].items():
            p.download_ptr(k, h.data_ptr(), VC)
        return dict(count=r["count"], residual=r["residual"], **st["down"])
    if kind == "host":
        for k, h in st["up"].items():
            p.upload_ptr(k, h.data_ptr(), VC)
        r = p.solve_rbgs(c["omega"], c["count"], c["eps"])
        p.download_ptr("X", st["x"].data_ptr(), VC)
        return dict(x=st["x"], count=r["count"], history=r["history"])
    p.fill("X", 0.0)
    if kind == "calls":
        r2 = []
        for _ in range(c["count"]):
            p.rbgs_sweep(c["omega"])
            r2.append(p.calc_r2())
        bb = p.dot("B", "B")
        p.exchange("X")
        return dict(x=_iterate(p, st["nb"]), r2=np.array(r2), bb=bb)
    if kind == "rbgs":
        r = p.solve_rbgs(c["omega"], c["count"], c["eps"])
    elif kind == "bicgstab":
        r = p.solve_bicgstab(c["omega"], c["pre"], c["count"], c["eps"], restart_drop=c["drop"])
    elif kind == "cg":
        r = p.solve_cg(c["omega"], c["pre"], c["count"], c["eps"])
    else:
        r = p.solve_mixed(omega=c["omega"], sweeps=c["sweeps"], sweeps_per_exchange=c["per"],
                          count_max=c["count"], epsilon=c["eps"], fp64_data=c["fp64"])
    return dict(x=_iterate(p, st["nb"]), count=r["count"], history=r["history"])


def work(case):
    """Bytes and flops per pass.  A block whose cells all have the same seven coefficients (no
    cut cell, no outer face) needs them once; the others need them per cell and pass."""
    grids = ([g for g, _ in _batch_problems(case, 0)] if case["kind"] == "batch" else [case])
    n = nn = 0
    for g in grids:
        level, index = _leaves(_key(g))
        n += len(level) * 4096
        nn += _varied_blocks(_key(g)) * 4096
    it, kind = case["count"], case["kind"]
    host = len(_leaves(_key(case))[0]) * W ** 3 * 8
    if kind == "calls":  # sweep, residual
        return dict(bytes=it * (40 * n + 112 * nn) + 16 * n, flops=it * 30 * n)
    if kind == "rbgs":  # x, b read, x written; residual and update of each cell
        return dict(bytes=it * (24 * n + 56 * nn), flops=it * 30 * n)
    if kind == "host":
        return dict(bytes=10 * host + it * (24 * n + 56 * nn), flops=it * 30 * n)
    if kind == "cg":  # Jacobi passes, p, A p, update
        k = case["pre"]
        per = 16 + 24 * (k - 1) + 24 + 16 + 48
        return dict(bytes=it * (per * n + 56 * (k + 1) * nn), flops=it * (16 * k + 24) * n)
    if kind in ("bicgstab", "step"):  # p and s with their first Jacobi pass, passes, A x, update
        k = case["pre"]
        per = 40 + 32 + 2 * 24 * (k - 1) + 2 * 24 + 64
        w = dict(bytes=it * (per * n + 56 * 2 * (k + 1) * nn), flops=it * (32 * k + 50) * n)
        if kind == "step":  # 4 host arrays each way; projections, exchange, assembly
            w["bytes"] += 8 * host + (57 * 2 + 24 + 49 + 112 + 14 * 8) * n
            w["flops"] += 200 * n
        return w
    passes = case["sweeps"] // case["per"]
    e, cw = (8, 56) if case.get("fp64") else (4, 28)
    per = (32 + e) + (24 + e) + 2 * (passes - 1) * (8 + 2 * e) + 2 * (16 + e) + 48 + 2 * e
    return dict(bytes=it * (per * n + (2 * passes * cw + 112) * nn),
                flops=it * (2 * case["sweeps"] * 15 + 60) * n)


# ---------------------------------------------------------------------------
# The path in plain torch, 64 bits, arrays [block][k][j][i]
# ---------------------------------------------------------------------------
def _key(case):
    return tuple(case[k] for k in ("level", "gx", "gy", "gz", "cx", "cy", "cz", "radius"))


def _box_distance2(key, L, idx):
    d2 = 0.0
    for a in range(3):
        lo = ORIGIN[a] + 4.0 / (1 << L) * idx[a]
        hi = lo + 4.0 / (1 << L)
        c = key[4 + a]
        d2 += max(lo - c, 0.0, c - hi) ** 2
    return d2


@functools.lru_cache(maxsize=None)
def _leaves(key):
    """(levels, indices) of the leaf blocks: refined within radius + 0.5 of the centre, 2:1
    balanced across faces, depth-first with x fastest."""
    top, root, reach2 = key[0], key[1:4], (key[7] + 0.5) ** 2
    branch = set()

    def build(L, x, y, z):
        if L < top and _box_distance2(key, L, (x, y, z)) <= reach2:
            branch.add((L, x, y, z))
            for c in range(8):
                build(L + 1, 2 * x + (c & 1), 2 * y + (c >> 1 & 1), 2 * z + (c >> 2))

    roots = [(x, y, z) for z in range(root[2]) for y in range(root[1]) for x in range(root[0])]
    for r in roots:
        build(0, *r)
    # a branch at level L >= 1 makes every face neighbour position at level L exist, so that
    # its children's neighbours are at most one level coarser
    todo = list(branch)
    while todo:
        L, x, y, z = todo.pop()
        if L == 0:
            continue
        for a in range(3):
            for d in (-1, 1):
                n = [x, y, z]
                n[a] += d
                if not 0 <= n[a] < root[a] << L:
                    continue
                l, p = L - 1, (n[0] >> 1, n[1] >> 1, n[2] >> 1)
                while l >= 0 and (l,) + p not in branch:
                    branch.add((l,) + p)
                    todo.append((l,) + p)
                    l, p = l - 1, (p[0] >> 1, p[1] >> 1, p[2] >> 1)
    lev, idx = [], []

    def emit(L, x, y, z):
        if (L, x, y, z) in branch:
            for c in range(8):
                emit(L + 1, 2 * x + (c & 1), 2 * y + (c >> 1 & 1), 2 * z + (c >> 2))
        else:
            lev.append(L)
            idx.append((x, y, z))

    for r in roots:
        emit(0, *r)
    return lev, idx


@functools.lru_cache(maxsize=None)
def _varied_blocks(key):
    """Blocks on the domain's surface or with the sphere's surface in them."""
    n = 0
    for L, id3 in zip(*_leaves(key)):
        near = _box_distance2(key, L, id3) <= key[7] ** 2
        far = sum(max(abs(ORIGIN[a] + 4.0 / (1 << L) * (id3[a] + s) - key[4 + a])
                      for s in (0, 1)) ** 2 for a in range(3)) >= key[7] ** 2
        edge = any(id3[a] == 0 or id3[a] == (key[1 + a] << L) - 1 for a in range(3))
        n += edge or (near and far)
    return n


def _dev(a, dtype=torch.float64):
    return torch.as_tensor(np.asarray(a)).to("cuda", dtype)


def _inputs(level, index, case, seed):
    """u*, cut distances, cut flags and fluid flags of every cell."""
    g = torch.Generator("cuda").manual_seed(int(seed))
    nb = len(level)
    shape = (nb, 16, 16, 16)
    dx = 4.0 / (2.0 ** _dev(level)) / 16.0
    out = {}
    for u, mean in zip(U_FIELDS, (1.0, 0.0, 0.0)):
        out[u] = mean + SIGMA * torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)
    D = []
    ar = torch.arange(16, device="cuda", dtype=torch.float64) + 0.5
    for a, c in enumerate((case["cx"], case["cy"], case["cz"])):
        org = ORIGIN[a] + dx * 16.0 * _dev(np.asarray(index).reshape(nb, 3)[:, a])
        p = org[:, None] + ar * dx[:, None] - c
        D.append(p.reshape((nb,) + ((1, 1, 16), (1, 16, 1), (16, 1, 1))[a]).expand(shape))
    gap = D[0] ** 2 + D[1] ** 2 + D[2] ** 2 - case["radius"] ** 2
    h = dx.reshape(nb, 1, 1, 1)
    for f in range(6):
        b = D[f // 2] * (1.0 if f & 1 else -1.0)
        disc = b * b - gap
        sq = disc.clamp(min=0.0).sqrt()
        t1, t2 = -b - sq, -b + sq
        ok1, ok2 = (t1 > 0) & (t1 <= h), (t2 > 0) & (t2 <= h)
        t = torch.where(ok1, t1, t2)
        cut = (disc >= 0) & (ok1 | ok2)
        d = (t / h).float().double().clamp(1e-6, 1.0)  # cut positions are 32-bit on input
        out["C%d" % f] = torch.where(cut, d, torch.ones_like(d))
        out["CID%d" % f] = cut.to(torch.int32)
    out["PID"] = (gap >= 0).to(torch.int32)
    return out


def _step_fields(level, index, case, seed):
    """A step's host arrays: u* and the last pressure, guide cells included."""
    g = torch.Generator("cuda").manual_seed(int(seed) + 7919)
    shape = (len(level), W, W, W)
    means = dict(zip(U_FIELDS + ("X",), (1.0, 0.0, 0.0, 0.0)))
    return {k: m + (0.02 if k == "X" else SIGMA) *
            torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)
            for k, m in means.items()}


def _axis_pos(f):
    """Interpolation cell (0-based) and weight of fine position f in [1, 32] of a coarse block."""
    i, r = f // 2, 0.25 + 0.5 * (f % 2)
    if f < 2:
        return 0, -0.25
    if f > 31:
        return 14, 1.25
    return i - 1, r


class _Path:
    """Guide cells, assembly, operator and solvers of one grid."""

    def __init__(self, case):
        lev, idx = _leaves(_key(case))
        self.lev, self.idx, self.nb = lev, idx, len(lev)
        self.root = (case["gx"], case["gy"], case["gz"])
        self.dx = 4.0 / (2.0 ** _dev(lev)) / 16.0
        at = {(L,) + tuple(i): n for n, (L, i) in enumerate(zip(lev, idx))}
        self.faces = [[self._face(at, n, f) for f in range(6)] for n in range(self.nb)]
        self.tables = {}
        k, j, i = torch.meshgrid(*[torch.arange(16, device="cuda")] * 3, indexing="ij")
        self.odd = (i + j + k) % 2 == 1

    def _face(self, at, n, f):
        L, id3, a = self.lev[n], list(self.idx[n]), f // 2
        id3[a] += 1 if f & 1 else -1
        if not 0 <= id3[a] < self.root[a] << L:
            return ("outer",)
        if (L,) + tuple(id3) in at:
            return ("same", at[(L,) + tuple(id3)])
        up = (L - 1,) + tuple(v >> 1 for v in id3)
        if up in at:
            return ("coarse", at[up], [v & 1 for v in self.idx[n]])
        t = [b for b in range(3) if b != a]
        fine = {}
        for q in range(4):
            c = [0, 0, 0]
            c[a] = 2 * id3[a] + (0 if f & 1 else 1)
            c[t[0]], c[t[1]] = 2 * id3[t[0]] + (q & 1), 2 * id3[t[1]] + (q >> 1)
            fine[q] = at[(L + 1,) + tuple(c)]
        return ("fine", fine)

    def _table(self, f, layer):
        """Guide cells of face f, layer 1 or 2: source cells, weights, and which are outer."""
        if (f, layer) in self.tables:
            return self.tables[f, layer]
        a, plus = f // 2, f & 1
        t = [b for b in range(3) if b != a]
        pats = {}

        def pattern(kind, so):
            if (kind, so) in pats:
                return pats[kind, so]
            src = np.zeros((256, 8), np.int64)
            wgt = np.zeros((256, 8))
            quad = np.zeros(256, np.int64)
            for p in range(256):
                tp = (p & 15, p >> 4)
                if kind in ("same", "outer"):
                    c = [0, 0, 0]
                    c[t[0]], c[t[1]] = tp
                    c[a] = ((layer - 1) if plus else 16 - layer) if kind == "same" else 15 * plus
                    src[p, 0], wgt[p, 0] = c[0] + 16 * (c[1] + 16 * c[2]), 1.0
                    continue
                lo, r = [0, 0, 0], [0.0, 0.0, 0.0]
                if kind == "coarse":
                    for s in range(2):
                        lo[t[s]], r[t[s]] = _axis_pos(tp[s] + 1 + 16 * so[t[s]])
                    lo[a], r[a] = _axis_pos(layer if plus else 33 - layer)
                else:
                    quad[p] = (tp[0] >> 3) + 2 * (tp[1] >> 3)
                    for s in range(2):
                        lo[t[s]] = 2 * (tp[s] & 7)
                    lo[a] = 2 * layer - 2 if plus else 16 - 2 * layer
                    r = [0.5, 0.5, 0.5]
                for m in range(8):
                    o = (m & 1, m >> 1 & 1, m >> 2)
                    c = [lo[b] + o[b] for b in range(3)]
                    src[p, m] = c[0] + 16 * (c[1] + 16 * c[2])
                    wgt[p, m] = math.prod(r[b] if o[b] else 1.0 - r[b] for b in range(3))
            pats[kind, so] = src, wgt, quad
            return pats[kind, so]

        src = np.zeros((self.nb, 256, 8), np.int64)
        wgt = np.zeros((self.nb, 256, 8))
        outer = np.zeros(self.nb, bool)
        for n in range(self.nb):
            face = self.faces[n][f]
            kind = face[0]
            s, w, quad = pattern(kind, tuple(face[2]) if kind == "coarse" else None)
            if kind == "fine":
                blk = np.array([face[1][q] for q in range(4)])[quad][:, None]
            else:
                blk = n if kind == "outer" else face[1]
            src[n], wgt[n], outer[n] = s + 4096 * blk, w, kind == "outer"
        self.tables[f, layer] = torch.as_tensor(src).cuda(), _dev(wgt), _dev(outer, torch.bool)
        return self.tables[f, layer]

    def guide(self, x, f, layer, bc):
        """[block][256] guide values across face f; bc: (types, values) per face."""
        src, wgt, outer = self._table(f, layer)
        g = (x.reshape(-1)[src] * wgt).sum(-1)
        v = bc[1][f]
        if bc[0][f] == ffvgpu.BC_DIRICHLET:
            o = 2.0 * v - g if layer == 1 else torch.full_like(g, v)
        else:
            o = g + (1.0 if f & 1 else -1.0) * layer * v * self.dx[:, None]
        return torch.where(outer[:, None], o, g)

    def guides(self, x, bc):
        return [self.guide(x, f, 1, bc).reshape(self.nb, 16, 16) for f in range(6)]

    @staticmethod
    def around(x, g):
        """The six neighbours of every cell: w, e, s, n, b, t."""
        return (torch.cat([g[0].unsqueeze(3), x[..., :-1]], 3),
                torch.cat([x[..., 1:], g[1].unsqueeze(3)], 3),
                torch.cat([g[2].unsqueeze(2), x[:, :, :-1]], 2),
                torch.cat([x[:, :, 1:], g[3].unsqueeze(2)], 2),
                torch.cat([g[4].unsqueeze(1), x[:, :-1]], 1),
                torch.cat([x[:, 1:], g[5].unsqueeze(1)], 1))

    def host(self, x, bc):
        """The host array of a field: interior and both guide layers of every face."""
        out = torch.zeros((self.nb, W, W, W), dtype=torch.float64, device="cuda")
        out[:, 2:18, 2:18, 2:18] = x
        for f in range(6):
            for layer in (1, 2):
                sl = [slice(None), slice(2, 18), slice(2, 18), slice(2, 18)]
                sl[3 - f // 2] = 17 + layer if f & 1 else 2 - layer
                out[tuple(sl)] = self.guide(x, f, layer, bc).reshape(self.nb, 16, 16)
        return out

    def assemble(self, inp, u, gu):
        """A (Ap, Aw..At) and b of the cut-cell pressure equation, outer faces folded in."""
        dx = self.dx.reshape(-1, 1, 1, 1)
        rho, vel = [None] * 6, [None] * 6
        for a in range(3):
            n = self.around(u[a], gu[a])
            vel[2 * a], vel[2 * a + 1] = 0.5 * (u[a] + n[2 * a]), 0.5 * (u[a] + n[2 * a + 1])
            rho[2 * a] = rho[2 * a + 1] = torch.full_like(u[a], 1.0 / RHOF)
        for a in range(3):
            m, p = 2 * a, 2 * a + 1
            for f, o in ((m, p), (p, m)):
                cut, d = inp["CID%d" % f] != 0, inp["C%d" % f]
                vel[f] = torch.where(cut, vel[o] * (d - 0.5) / (d + 0.5), vel[f])
                rho[o] = torch.where(cut, (1.0 / RHOF) / (d + 0.5), rho[o])
                rho[f] = torch.where(cut, torch.zeros_like(d), rho[f])
            both = (inp["CID%d" % m] != 0) & (inp["CID%d" % p] != 0)
            for f in (m, p):
                vel[f] = torch.where(both, torch.zeros_like(dx), vel[f])
                rho[f] = torch.where(both, torch.zeros_like(dx), rho[f])
        fluid = inp["PID"] == 1
        A = [None] + [torch.where(fluid, r / (dx * dx), torch.ones_like(dx)) for r in rho]
        A[0] = torch.where(fluid, -sum(A[1:]), torch.full_like(dx, -6.0))
        div = sum(vel[2 * a + 1] - vel[2 * a] for a in range(3)) / dx
        b = torch.where(fluid, div / DT, torch.zeros_like(dx))
        for f in range(6):
            outer = self._table(f, 1)[2]
            sl = [slice(None)] * 4
            sl[3 - f // 2] = 15 if f & 1 else 0
            af = A[1 + f][tuple(sl)] * outer[:, None, None]
            A[0][tuple(sl)] += -af if ffvgpu.P_BC_TYPE[f] == ffvgpu.BC_DIRICHLET else af
            A[1 + f][tuple(sl)] -= af
        return A, b

    def project(self, inp, p, gp, u, sign):
        """u + sign dt grad p / rho, 0 in solid cells."""
        dx = self.dx.reshape(-1, 1, 1, 1)
        n = self.around(p, gp)
        fluid = inp["PID"] == 1
        out, faces = [], []
        for a in range(3):
            g = [(p - n[2 * a]) / dx / RHOF, (n[2 * a + 1] - p) / dx / RHOF]
            c = [inp["CID%d" % f] != 0 for f in (2 * a, 2 * a + 1)]
            d = [inp["C%d" % f] for f in (2 * a, 2 * a + 1)]
            g[0] = torch.where(c[0], g[1] * (d[0] - 0.5) / (d[0] + 0.5), g[0])
            g[1] = torch.where(c[1], g[0] * (d[1] - 0.5) / (d[1] + 0.5), g[1])
            g = [torch.where(c[0] & c[1], torch.zeros_like(v), v) for v in g]
            out.append(torch.where(fluid, u[a] + sign * 0.5 * (g[0] + g[1]) * DT,
                                   torch.zeros_like(p)))
        return out

    def apply(self, x, g=None):
        n = self.around(x, g if g is not None else self.guides(x, P_BC))
        return sum(a * v for a, v in zip(self.A[1:], n)) + self.A[0] * x

    def jacobi(self, rhs, omega, passes):
        z = torch.zeros_like(rhs)
        for k in range(passes):
            off = self.apply(z) - self.A[0] * z if k else 0.0
            z = z - omega * (z - (rhs - off) / self.A[0])
        return z

    def sweep(self, x, omega, g):
        for c in (0, 1):
            off = sum(a * v for a, v in zip(self.A[1:], self.around(x, g)))
            new = x - omega * (x - (self.b - off) / self.A[0])
            x = torch.where(self.odd if c else ~self.odd, new, x)
        return x

    def residual(self, r, bb):
        rr = float((r * r).sum())
        return math.sqrt(rr / bb) if bb > np.finfo(np.float32).tiny else math.sqrt(rr)

    def rbgs(self, x, g, omega, count, eps):
        bb, hist = float((self.b * self.b).sum()), []
        for n in range(1, count + 1):
            x = self.sweep(x, omega, g)
            g = self.guides(x, P_BC)
            hist.append(self.residual(self.b - self.apply(x, g), bb))
            if hist[-1] <= eps:
                return x, n, hist
        return x, count + 1, hist

    def cg(self, x, g, omega, pre, count, eps):
        bb, hist, rr0, p = float((self.b * self.b).sum()), [], 1.0, None
        r = self.b - self.apply(x, g)
        for n in range(1, count + 1):
            z = self.jacobi(r, omega, pre)
            rr1 = float((r * z).sum())
            p = z if p is None else z + rr1 / rr0 * p
            q = self.apply(p)
            alpha = rr1 / float((q * p).sum())
            x, r, rr0 = x + alpha * p, r - alpha * q, rr1
            hist.append(self.residual(r, bb))
            if hist[-1] <= eps:
                return x, n, hist
        return x, count + 1, hist

    def bicgstab(self, x, g, omega, pre, count, eps, drop):
        bb, hist, p, q = float((self.b * self.b).sum()), [], None, None
        r = self.b - self.apply(x, g)
        at, fresh = (self.residual(r, bb) * drop if drop > 0 else -1.0), True
        for n in range(1, count + 1):
            if fresh:
                r0, rr0, alpha, gamma = r, 1.0, 0.0, 1.0
            rr1 = float((r * r0).sum())
            p = r if fresh else r + rr1 / rr0 * alpha / gamma * (p - gamma * q)
            ph = self.jacobi(p, omega, pre)
            q = self.apply(ph)
            alpha = rr1 / float((q * r0).sum())
            s = r - alpha * q
            sh = self.jacobi(s, omega, pre)
            t = self.apply(sh)
            gamma = float((t * s).sum()) / float((t * t).sum())
            x, r, rr0, fresh = x + alpha * ph + gamma * sh, s - gamma * t, rr1, False
            hist.append(self.residual(r, bb))
            if hist[-1] <= eps:
                return x, n, hist
            if 0 < at and hist[-1] <= at:
                at, fresh = hist[-1] * drop, True
        return x, count + 1, hist


P_BC = (ffvgpu.P_BC_TYPE, ffvgpu.P_BC_VALUE)


def _device_layout(x):
    """[nb][16][16][16] -> [nb][4096] as the pool holds it: cells by colour, then k, j, i/2."""
    k, j, i = np.meshgrid(*[np.arange(16)] * 3, indexing="ij")
    slot = (((i + j + k) & 1) << 11) | ((k * 16 + j) << 3) | (i >> 1)
    at = np.empty(4096, np.int64)
    at[slot.reshape(-1)] = np.arange(4096)
    return x.reshape(-1, 4096)[:, torch.as_tensor(at).cuda()]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mixed", "batch"):
        return None  # a cut-off iterate of a preconditioner on rounded data has no such value
    nb = len(_leaves(_key(case))[0])
    if nb * case["count"] * COST.get(kind, 5) > 5_000_000:
        return None  # over about 20 seconds
    P = _Path(case)
    inp = _inputs(P.lev, P.idx, case, seed)
    u = [inp[k] for k in U_FIELDS]
    ubc = [(ffvgpu.U_BC_TYPE, ffvgpu.U_BC_VALUE[k]) for k in U_FIELDS]
    f, x0 = None, torch.zeros_like(u[0])
    g0 = [torch.zeros_like(x0[:, 0])] * 6
    if kind == "step":
        f = _step_fields(P.lev, P.idx, case, seed)
        mid, X = slice(2, 18), f["X"]
        x0 = X[:, mid, mid, mid]
        g0 = [X[:, mid, mid, 1], X[:, mid, mid, 18], X[:, mid, 1, mid], X[:, mid, 18, mid],
              X[:, 1, mid, mid], X[:, 18, mid, mid]]
        u = P.project(inp, x0, g0, [f[k][:, mid, mid, mid] for k in U_FIELDS], 1.0)
    P.A, P.b = P.assemble(inp, u, [P.guides(v, bc) for v, bc in zip(u, ubc)])
    if kind == "calls":
        x, g, r2 = x0, g0, []
        for _ in range(case["count"]):
            x = P.sweep(x, case["omega"], g)
            g = P.guides(x, P_BC)
            r2.append(float(((P.b - P.apply(x, g)) ** 2).sum()))
        return dict(x=_device_layout(x), r2=np.array(r2), bb=float((P.b * P.b).sum()))
    if kind in ("rbgs", "host"):
        x, n, hist = P.rbgs(x0, g0, case["omega"], case["count"], case["eps"])
    elif kind == "cg":
        x, n, hist = P.cg(x0, g0, case["omega"], case["pre"], case["count"], case["eps"])
    else:
        x, n, hist = P.bicgstab(x0, g0, case["omega"], case["pre"], case["count"], case["eps"],
                                case["drop"])
    if kind == "step":
        u = P.project(inp, x, P.guides(x, P_BC), u, -1.0)
        out = {k: P.host(v, bc).cpu() for k, v, bc in zip(U_FIELDS, u, ubc)}
        return dict(count=n, residual=hist[-1], X=P.host(x, P_BC).cpu(), **out)
    if kind == "host":
        return dict(x=P.host(x, P_BC).cpu(), count=n, history=np.array(hist))
    return dict(x=_device_layout(x), count=n, history=np.array(hist))
