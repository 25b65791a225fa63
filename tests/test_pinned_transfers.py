"""Downloads into pinned arrays that start anywhere in a line, for rows shorter and longer than the pieces a
warp writes, against downloads into pageable ones; nothing beside the array is written.  Which arrays count as
pinned: those that registrations cover from end to end."""
import ctypes as C

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


def test_an_array_is_pinned_only_where_ranges_cover_it():
    from test_device_math_host import LIB
    lib = C.CDLL(LIB)
    lib.hm_host_covered.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_uint64, C.c_uint64]

    def covered(p, size, *ranges):
        r = np.array(ranges, np.uint64).reshape(-1, 2)
        b, s = np.ascontiguousarray(r[:, 0]), np.ascontiguousarray(r[:, 1])
        return bool(lib.hm_host_covered(b.ctypes.data, s.ctypes.data, len(r), p, size))

    page = 4096
    one, two, far = (page, 2 * page), (3 * page, page), (5 * page, page)
    assert covered(page, 2 * page, one) and covered(page + 8, 8, one)
    assert covered(page + 8, 3 * page - 8, one, two)                # next to each other
    assert covered(page, 3 * page, two, one)
    assert not covered(page, 4 * page + 8, one, two, far)           # a page between them is in none
    assert not covered(3 * page, 3 * page, one, two, far)           # both ends are
    assert not covered(page - 8, 16, one) and not covered(3 * page - 8, 16, one)
    assert not covered(0, 8) and not covered(page, 0, one)
    assert not covered(2 ** 64 - 8, 16, (2 ** 64 - page, page - 1))


@pytest.mark.gpu
def test_an_array_over_two_registrations():
    import torch
    from hyperflow_gb300 import CartSolver, cases
    rt = torch.cuda.cudart()
    a, b = (CartSolver(cases.quadrant_case(100, cfl=cases.CFL_2D)) for _ in range(2))
    want = a.state(0)
    page, size = 65536, want.nbytes
    assert page < size < 6 * page
    raw = np.zeros(8 * page, np.uint8)
    base = (raw.ctypes.data + page - 1) // page * page
    at = base - raw.ctypes.data + page - 8                          # 8 bytes in the first, the rest in the second
    U = raw[at:at + size].view(np.float64).reshape(want.shape)
    assert not CartSolver.host_mapped(U)
    for start, length in ((base, page), (base + page, 6 * page)):
        assert int(rt.cudaHostRegister(start, length, 0)) == 0
    try:
        assert CartSolver.host_mapped(U)
        U[...] = want * 1.01
        a.set_state(0, U)
        b.set_state(0, U.copy())
        assert a.step() == b.step()
        np.testing.assert_array_equal(a.state(0, out=U), b.state(0))
    finally:
        for start in (base, base + page):
            rt.cudaHostUnregister(start)
    assert not CartSolver.host_mapped(U)
