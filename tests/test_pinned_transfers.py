"""Downloads into pinned arrays that start anywhere in a line, for rows shorter and longer than the pieces a
warp writes, against downloads into pageable ones; nothing beside the array is written."""
import numpy as np
import pytest


def _pinned(n):
    import torch
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1, 15, 16, 31])
@pytest.mark.parametrize("nx,ny", [(4, 4), (29, 7), (30, 8), (31, 9), (125, 4), (126, 33), (129, 5), (257, 130)])
def test_pinned_download_equals_pageable_at_any_offset(nx, ny, offset):
    from hyperflow_gb300 import CartSolver, cases
    for scheme, limiter in (("Godunov", None), ("MUSCLHancock", "MinBee")):
        s = CartSolver(cases.quadrant_case(nx, ny=ny, scheme=scheme, limiter=limiter, cfl=cases.CFL_2D))
        s.run(2)
        want = s.state(0)
        buf = _pinned(want.size + 64)
        buf[...] = -1.0
        got = buf[offset:offset + want.size].reshape(want.shape)
        assert CartSolver.host_mapped(got)
        np.testing.assert_array_equal(s.state(0, out=got), want)
        assert (buf[:offset] == -1.0).all() and (buf[offset + want.size:] == -1.0).all()
        s.close()
