"""Divisions by a uniform block's diagonal, which the stencil kernels form from
one reciprocal where that cannot under- or overflow and leave to '/' elsewhere:
diagonals of arbitrary mantissa, a different one in every block, exponents on
both sides of the fast form's bounds, right-hand sides that are zero over whole
blocks or far from 1.  Bit equality with the oracle for every solver that
divides: the RBGS pass, the Jacobi pass and the one from zero."""
import numpy as np
import pytest

from helpers import VC, device_problem, problem
from test_gpu_varied import COEFS, run

pytestmark = pytest.mark.gpu

SOLVERS = [("rbgs", (1.1, 3, 0.0)), ("cg", (1.0, 1, 3, 0.0)), ("cg", (0.9, 3, 3, 0.0)),
           ("bicgstab", (1.0, 2, 3, 0.0))]


def compare(solver, args, scale=1.0, b_scale=1.0, zero=False):
    g, inp, O = problem(2)
    P = device_problem(g, inp)
    rng = np.random.default_rng(8)
    for f in COEFS:
        base = -6.5 if f == "AP" else 1.0
        a = np.broadcast_to(base * rng.uniform(0.9, 1.9, (g.nb, 1, 1, 1)) * scale,
                            (g.nb, 20, 20, 20)).copy()
        P.upload(f, a, VC)
        O.field(f)[...] = a
    b = rng.standard_normal((g.nb, 20, 20, 20)) * b_scale
    if zero:
        b[::2] = 0.0
        b[1::4] *= -0.0
    P.upload("B", b, VC)
    O.field("B")[...] = b
    run(g, P, O, solver, args)
    P.close()
    O.close()


@pytest.mark.parametrize("solver,args", SOLVERS)
@pytest.mark.parametrize("exponent", [0, -248, -253, -300, 247, 252, 300])
def test_diagonals_around_the_bounds(solver, args, exponent):
    s = 2.0 ** exponent
    compare(solver, args, scale=s, b_scale=max(1.0, s))


@pytest.mark.parametrize("solver,args", SOLVERS)
@pytest.mark.parametrize("b_scale,zero", [(1.0, True), (1e140, False), (1e-15, True)])
def test_right_hand_sides(solver, args, b_scale, zero):
    compare(solver, args, b_scale=b_scale, zero=zero)
