"""Solves on a device that is nearly full: room for the solver's vectors but not
for the guide buffers, without which the same solve runs."""
import numpy as np
import pytest
import torch
from cuda.bindings import runtime as cudart

from helpers import VC, assert_bitwise, device_problem, interior, problem

pytestmark = pytest.mark.gpu

MB = 1 << 20


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def fill_up(leave):
    """Allocations after which at most 'leave' bytes are free, in granules of 2 MB."""
    hog, size = [], (free_bytes() - leave) // (2 * MB) * (2 * MB)
    while free_bytes() > leave:
        err, p = cudart.cudaMalloc(size)
        if err == cudart.cudaError_t.cudaSuccess:
            hog.append(p)
            size = max(2 * MB, (free_bytes() - leave) // (2 * MB) * (2 * MB))
        else:
            cudart.cudaGetLastError()
            size = size // 2 // (2 * MB) * (2 * MB)
            assert size, "no granule left"
    return hog


@pytest.mark.parametrize("solver,args", [("rbgs", (1.0, 6, 0.0)), ("cg", (1.0, 2, 6, 0.0)),
                                         ("bicgstab", (1.0, 2, 6, 0.0))])
def test_solve_without_room_for_the_guide_buffers(solver, args):
    g, inp, O = problem(3)
    torch.cuda.empty_cache()
    P = device_problem(g, inp)
    P.fill("X", 0.0)
    P.solve_bicgstab(1.0, 0, 2, 0.0)  # the kernels without pushed guides are loaded
    P.close()
    P = device_problem(g, inp)
    P.fill("X", 0.0)
    before = free_bytes()
    ref = getattr(P, "solve_" + solver)(*args)
    need = before - free_bytes()
    x = interior(P.download("X", VC)).copy()
    P.close()
    guides = 2 * g.nb * 6 * 256 * 8
    assert need > guides
    P = device_problem(g, inp)
    P.fill("X", 0.0)
    hog = fill_up(need - guides // 2)
    try:
        r = getattr(P, "solve_" + solver)(*args)
    finally:
        for p in hog:
            cudart.cudaFree(p)
    assert_bitwise(r["history"], ref["history"], "history")
    assert_bitwise(interior(P.download("X", VC)), x, "x")
    assert np.isfinite(x).all()
    P.close()
    O.close()
