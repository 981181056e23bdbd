"""Uploads in every layout the pack kernel reads: guide widths 1 to 4 (runs of
rows of other lengths), buffers 16-byte aligned and only 8-byte aligned (pairs
of values or single ones per load), pageable and pinned, fields with and
without guide cells.  The values must reach the same cells as in the
reference width of 2: interiors are compared after a download, the stored
guide layer through a sweep that reads it."""
import numpy as np
import pytest
import torch

import ffvgpu
from helpers import VC, assert_bitwise, device_problem, interior, problem

pytestmark = pytest.mark.gpu


def relaid(a, vc, rng):
    """a (width VC) at width vc: interior and first guide layer kept, the rest noise."""
    w = 16 + 2 * vc
    out = rng.standard_normal((a.shape[0], w, w, w))
    out[:, vc - 1:vc + 17, vc - 1:vc + 17, vc - 1:vc + 17] = a[:, 1:19, 1:19, 1:19]
    return out


@pytest.mark.parametrize("vc", [1, 2, 3, 4])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("pinned", [False, True])
def test_upload_layouts(vc, offset, pinned):
    g, inp, O = problem(1)
    P = device_problem(g, inp)
    rng = np.random.default_rng(5)
    x = rng.standard_normal((g.nb, 20, 20, 20))
    ap = P.download("AP", VC)
    P.upload("X", x, VC)
    P.rbgs_sweep(1.1)
    ref = P.download("X", VC)
    for field, a in (("X", x), ("AP", ap)):
        r = relaid(a, vc, rng)
        buf = torch.empty(r.size + 2, dtype=torch.float64, pin_memory=pinned)
        start = offset + (buf.data_ptr() // 8) % 2  # element 'start' is 8 bytes off a 16-byte line
        view = buf[start:start + r.size]
        view.copy_(torch.from_numpy(r.reshape(-1)))
        assert (view.data_ptr() % 16 == 0) == (offset == 0)
        P.upload_ptr(field, view.data_ptr(), vc)
        if field == "X":
            assert_bitwise(interior(P.download("X", VC)), interior(x), "x interior")
            P.rbgs_sweep(1.1)
            assert_bitwise(P.download("X", VC), ref, "x after a sweep")
        else:
            assert_bitwise(interior(P.download("AP", VC)), interior(ap), "Ap interior")
    P.close()
    O.close()
