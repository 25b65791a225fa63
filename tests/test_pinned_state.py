"""State uploads and downloads of pinned arrays (kernels over the host link) against pageable ones (copies):
the same device state, TimeStep and steps, for widths around a warp's 32 cells and blocks of one and
two ghost layers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pinned(shape):
    import torch
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


@pytest.mark.parametrize("nx,ny", [(4, 4), (28, 5), (31, 9), (33, 40), (127, 3), (257, 66)])
@pytest.mark.parametrize("scheme", ["Godunov", "MUSCLHancock"])
def test_pinned_state_equals_pageable(scheme, nx, ny):
    from hyperflow_gb300 import CartSolver, cases
    ny = max(ny, 4)
    case = cases.quadrant_case(nx, ny=ny, scheme=scheme, limiter="MinBee" if scheme == "MUSCLHancock" else None,
                               cfl=cases.CFL_2D)
    a, b = CartSolver(case), CartSolver(case)
    U = a.state(0)
    U = U * (1.0 + 0.01 * np.random.default_rng(nx).random(U.shape[1:]))
    P = _pinned(U.shape)
    P[...] = U
    assert CartSolver.host_mapped(P) and not CartSolver.host_mapped(U)
    a.set_state(0, U)
    b.set_state(0, P)
    for steps in (0, 3, 4):
        a.run(steps)
        b.run(steps)
        assert a.time() == b.time()
        got = _pinned(U.shape)
        got[...] = -1.0
        np.testing.assert_array_equal(b.state(0, out=got), a.state(0))
    np.testing.assert_array_equal(P, U)
