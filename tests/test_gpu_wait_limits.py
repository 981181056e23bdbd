"""Bounded waits of the FP64 stencil kernels that run out on the device, without
faulting it: a test hook leaves one copy out, so that the wait for it gives up
after a short limit in the middle of a CTA's blocks.  The solve must end with
FFVGPU_TIMEOUT, the copies that are in flight must be waited for (no 'drain' in
the message), and the same pool must then solve bit for bit as the oracle."""
import numpy as np
import pytest

import ffvgpu
from helpers import VC, assert_bitwise, device_problem, interior, problem
from test_gpu_varied import run, set_varied

pytestmark = pytest.mark.gpu


def times_out(P, solve, *words):
    P.fill("X", 0.0)
    P.set_wait_limit(0.05)
    with pytest.raises(ffvgpu.FFVGPUError) as e:
        solve()
    P.set_wait_limit(4.0)
    assert e.value.status == ffvgpu.TIMEOUT
    assert "drain" not in str(e.value)
    for w in words:
        assert w in str(e.value)


# one block a CTA; a CTA's second block; a block handed out; the coefficient ring
@pytest.mark.parametrize("level,kw,varied", [(2, {}, None), (0, dict(root_grid=(9, 6, 6)), None),
                                             (4, {}, None), (3, {}, 1.0)])
@pytest.mark.parametrize("count", [1, 6])
def test_rbgs_wait_runs_out(level, kw, varied, count):
    g, inp, O = problem(level, **kw)
    P = device_problem(g, inp)
    if varied is not None:
        set_varied(g, P, O, varied)
    P.stall_next_solve()
    times_out(P, lambda: P.solve_rbgs(1.1, count, 0.0), "consumer")
    run(g, P, O, "rbgs", (1.1, count, 0.0))
    P.close()
    O.close()


# one block a CTA; two; blocks of a list's third chunk (one CTA); the coefficient ring
@pytest.mark.parametrize("level,ctas,varied", [(2, 0, None), (3, 0, None), (3, 1, None),
                                               (3, 0, 1.0)])
@pytest.mark.parametrize("solver,args", [("cg", (1.0, 1, 4, 0.0)), ("cg", (1.0, 3, 4, 0.0)),
                                         ("bicgstab", (1.0, 1, 4, 0.0)),
                                         ("bicgstab", (1.0, 2, 4, 0.0))])
def test_krylov_stencil_wait_runs_out(level, ctas, varied, solver, args):
    g, inp, O = problem(level)
    P = device_problem(g, inp)
    if varied is not None:
        set_varied(g, P, O, varied)
    P.cap_grids(ctas)
    P.stall_next_matvec()
    times_out(P, lambda: getattr(P, "solve_" + solver)(*args),
              "A*x" if varied else "FP64 A*x or Jacobi pass")
    run(g, P, O, solver, args)
    P.close()
    O.close()
