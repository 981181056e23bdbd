"""Pools in which most blocks' coefficients vary from cell to cell (variable
density, cells cut everywhere), where the FP64 solvers run on the kernels that
stream the coefficients through a ring: bit equality with the oracle on both
sides of the rule's line, with uniform blocks among the varied ones, and when
an upload of A moves a pool from one side to the other."""
import numpy as np
import pytest

import ffvgpu
from helpers import VC, assert_bitwise, device_problem, interior, problem

pytestmark = pytest.mark.gpu

COEFS = ("AP", "AW", "AE", "AS", "AN", "AB", "AT")


def set_varied(g, P, O, share, seed=3):
    """A share of the blocks gets coefficients that differ in every cell, the others one
    coefficient set each."""
    rng = np.random.default_rng(seed)
    varied = np.zeros((g.nb, 1, 1, 1), bool)
    varied[rng.permutation(g.nb)[:round(share * g.nb)]] = True
    for f in COEFS:
        base = -6.5 if f == "AP" else 1.0
        a = base * (1.0 + 0.01 * rng.uniform(-1.0, 1.0, (g.nb, 20, 20, 20)))
        a = np.where(varied, a, a[:, 10:11, 10:11, 10:11])
        P.upload(f, a, VC)
        O.field(f)[...] = a


def run(g, P, O, solver, args):
    P.fill("X", 0.0)
    O.field("X")[...] = 0.0
    ro = getattr(O, "solve_" + solver)(*args)
    rg = getattr(P, "solve_" + solver)(*args)
    assert rg["count"] == ro["count"]
    assert_bitwise(rg["history"], ro["history"], "history")
    assert_bitwise(interior(P.download("X", VC)), interior(O.field("X")), "x")


@pytest.mark.parametrize("root,share", [((9, 6, 6), 1.0), ((37, 4, 2), 1.0), ((11, 9, 3), 1.0),
                                        ((9, 6, 6), 0.9), ((10, 9, 9), 0.5), ((10, 9, 9), 0.3)])
@pytest.mark.parametrize("solver,args", [("cg", (1.0, 1, 3, 0.0)), ("cg", (1.0, 3, 3, 0.0)),
                                         ("bicgstab", (1.0, 1, 3, 0.0)),
                                         ("bicgstab", (0.9, 3, 3, 0.0))])
def test_krylov_on_varied_pools(root, share, solver, args):
    g, inp, O = problem(0, root_grid=root, radius=0.5)
    P = device_problem(g, inp)
    set_varied(g, P, O, share)
    run(g, P, O, solver, args)
    P.close()
    O.close()


@pytest.mark.parametrize("root,share", [((9, 6, 6), 1.0), ((37, 4, 2), 1.0), ((11, 9, 3), 1.0),
                                        ((9, 6, 6), 0.95), ((10, 9, 9), 0.5), ((10, 9, 9), 0.3)])
@pytest.mark.parametrize("solver,args", [("rbgs", (1.1, 1, 0.0)), ("rbgs", (1.1, 6, 0.0)),
                                         ("rbgs_fixed_average", (1.0, None, 3, 0.0))])
def test_rbgs_on_varied_pools(root, share, solver, args):
    g, inp, O = problem(0, root_grid=root, radius=0.5)
    P = device_problem(g, inp)
    set_varied(g, P, O, share)
    run(g, P, O, solver, args)
    P.close()
    O.close()


def test_single_rbgs_calls_on_a_varied_pool():
    """Stored guides as uploaded, then as the sweep's exchange left them; the early stop of a
    solve with a criterion; a wait limit of 0 ends in TIMEOUT and leaves the pool usable."""
    g, inp, O = problem(3)
    P = device_problem(g, inp)
    set_varied(g, P, O, 0.9)
    x = np.random.default_rng(4).standard_normal((g.nb, 20, 20, 20))
    P.upload("X", x, VC)
    O.field("X")[...] = x
    for _ in range(2):
        assert P.calc_r2() == O.calc_r2()
        P.rbgs_sweep(1.2)
        O.rbgs_sweep(1.2)
        O.exchange("X", ffvgpu.P_BC_TYPE, ffvgpu.P_BC_VALUE)
        assert_bitwise(interior(P.download("X", VC)), interior(O.field("X")), "x")
    run(g, P, O, "rbgs", (1.2, 200, 0.02))
    P.set_wait_limit(0.0)
    with pytest.raises(ffvgpu.FFVGPUError) as e:
        P.solve_rbgs(1.2, 5, 0.0)
    assert e.value.status == ffvgpu.TIMEOUT and "drain" not in str(e.value)
    P.set_wait_limit(4.0)
    run(g, P, O, "rbgs", (1.2, 5, 0.0))
    P.close()
    O.close()


@pytest.mark.parametrize("solver,args", [("cg", (1.0, 2, 4, 0.0)), ("bicgstab", (1.0, 2, 4, 0.0)),
                                         ("rbgs", (1.0, 7, 0.0))])
def test_coefficients_replaced_between_solves(solver, args):
    """2:1 faces (level 3), A replaced between solves so that the pool changes sides twice, and
    grids capped to one CTA."""
    g, inp, O = problem(3)
    P = device_problem(g, inp)
    for share in (1.0, 0.0, 0.8):
        set_varied(g, P, O, share)
        run(g, P, O, solver, args)
    P.cap_grids(1)
    run(g, P, O, solver, args)
    P.close()
    O.close()
