"""The RBGS pass where its launch and its arithmetic change form: block counts
around one and two blocks per SM (and one block alone), where the grid deals
out further blocks as CTAs free up; and right-hand sides whose quotients the
fast division by a uniform block's diagonal must leave to '/' (zeros, values
near the ends of the exponent range, infinities).  Bit equality with the
oracle throughout."""
import numpy as np
import pytest

import ffvgpu
from helpers import VC, assert_bitwise, device_problem, interior, problem

pytestmark = pytest.mark.gpu


def compare(g, inp, O, count, scale=None):
    P = device_problem(g, inp)
    if scale is not None:
        with np.errstate(all="ignore"):
            b = P.download("B", VC) * scale
        P.upload("B", b, VC)
        O.field("B")[...] = b
    P.fill("X", 0.0)
    O.field("X")[...] = 0.0
    ro = O.solve_rbgs(1.1, count, 0.0)
    rg = P.solve_rbgs(1.1, count, 0.0)
    assert_bitwise(rg["history"], ro["history"], "history")
    assert_bitwise(interior(P.download("X", VC)), interior(O.field("X")), "x")
    P.close()
    O.close()


@pytest.mark.parametrize("level,root,radius", [
    (0, (1, 1, 1), 0.5), (0, (37, 4, 1), 0.5), (0, (149, 1, 1), 0.5), (0, (37, 8, 1), 0.5),
    (0, (27, 11, 1), 0.5), (0, (8, 8, 8), 3.0), (2, (3, 2, 2), 0.9), (4, (4, 2, 2), 0.55)])
def test_block_counts(level, root, radius):
    compare(*problem(level, root_grid=root, radius=radius), 4)


@pytest.mark.parametrize("scale", [0.0, -0.0, 1e-310, 1e-290, 1e-200, 1e200, 1e290, np.inf])
def test_quotients_at_the_ends_of_the_range(scale):
    compare(*problem(2), 3, scale)


@pytest.mark.parametrize("solver", ["rbgs", "cg", "bicgstab", "mixed", "mixed 1 pass", "mixed 4 passes"])
def test_one_sided_neighbour_table(solver):
    """Guides are pushed to neighbours only where every face record is matched by the
    neighbour's; with a block that names a neighbour which does not name it (it has the
    identity for A and b = 0, so it adds zeros to every sum), the solves take all guides from
    the neighbours' interiors: the same bits."""
    g, inp, O = problem(2)
    P = device_problem(g, inp)
    kind, ids = g.neighbors()
    n = g.nb + 1
    kind = np.concatenate([kind, np.zeros((1, 6), np.int32)])
    ids = np.concatenate([ids, np.full((1, 6, 4), -1, np.int32)])
    kind[-1, 0], ids[-1, 0, 0] = ffvgpu.NB_SAME, 0
    level = np.concatenate([g.level, g.level[:1]])
    index = np.concatenate([g.index, g.index[:1]]).reshape(-1)
    d = g.desc()
    d.num_blocks = n
    d.level, d.block_index = level.ctypes.data, index.ctypes.data
    d.neighbor_kind, d.neighbor_ids = kind.ctypes.data, ids.ctypes.data
    Q = ffvgpu.Pool(d)
    for f in ("AP", "AW", "AE", "AS", "AN", "AB", "AT", "B"):
        a = P.download(f, VC)
        Q.upload(f, np.concatenate([a, np.full_like(a[:1], 1.0 if f == "AP" else 0.0)]), VC)
    r = []
    for p in (P, Q):
        p.fill("X", 0.0)
        r.append(p.solve_rbgs(1.0, 8, 0.0) if solver == "rbgs" else
                 p.solve_cg(1.0, 3, 8, 0.0) if solver == "cg" else
                 p.solve_bicgstab(1.0, 2, 8, 0.0) if solver == "bicgstab" else
                 p.solve_mixed(1.5, 8, {"mixed": 4, "mixed 1 pass": 8}.get(solver, 2), 6, 0.0))
    assert_bitwise(r[1]["history"], r[0]["history"], "history")
    assert_bitwise(interior(Q.download("X", VC))[:g.nb], interior(P.download("X", VC)), "x")
    P.close()
    Q.close()
    O.close()
