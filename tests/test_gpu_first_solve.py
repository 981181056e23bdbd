"""A pool's first solve is mostly device allocations on small grids, each a
tenth of a millisecond or more: the solvers' vectors, their tables and the
pushed guides come as one allocation each."""
import pytest
from torch.profiler import ProfilerActivity, profile

from helpers import device_problem, problem

pytestmark = pytest.mark.gpu


def allocations(f):
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        f()
    names = [e.name for e in p.events()]
    assert any(n.startswith("cudaLaunchKernel") for n in names)  # the library's calls are seen
    return sum(n == "cudaMalloc" for n in names)


# the solvers' tables, the pushed guides and the residual history; the Krylov vectors
@pytest.mark.parametrize("solver,args,most", [("rbgs", (1.0, 3, 0.0), 3), ("cg", (1.0, 2, 3, 0.0), 4),
                                              ("bicgstab", (1.0, 2, 3, 0.0), 4)])
def test_first_solve_allocations(solver, args, most):
    g, inp, O = problem(2)
    P = device_problem(g, inp)
    P.fill("X", 0.0)
    P.dot("X", "X")
    solve = lambda: getattr(P, "solve_" + solver)(*args)  # noqa: E731
    n = allocations(solve)
    assert 1 <= n <= most, n
    assert allocations(solve) == 0
    P.close()
    O.close()
