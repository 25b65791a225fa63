"""A step of one block in one launch (no ghost fill kernel) against the oracle and against the path with
the fill: every kind of side, blocks of a tile and of a cell past a tile's edge, the end-time clamp, and
changes of path between runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(nx, ny, scheme, sides, t_end=1.0e9):
    from hyperflow_gb300 import cases
    case = cases.quadrant_case(nx, ny=ny, scheme=scheme, limiter="VanLeer" if scheme == "MUSCLHancock" else None,
                               cfl=cases.CFL_2D, t_end=t_end)
    flow = {"type": "Dirichlet", "variables": "Primitive", "flow_state": [1.1, 2.5, 0.3, 1.2]}
    kinds = {"T": {"type": "Transmissive"}, "R": {"type": "Reflective"}, "D": flow}
    case["mesh"]["blocks"][0]["boundaries"] = {s: kinds[k] for s, k in zip(("bottom", "right", "top", "left"), sides)}
    return case


@pytest.mark.parametrize("sides", ["TTTT", "RRRR", "RTRD", "DDDD", "TRDT"])
@pytest.mark.parametrize("scheme,nx,ny", [("Godunov", 5, 4), ("Godunov", 33, 23), ("Godunov", 97, 65),
                                          ("MUSCLHancock", 4, 5), ("MUSCLHancock", 33, 19), ("MUSCLHancock", 65, 41)])
def test_one_launch_step_equals_oracle(port_lib, scheme, nx, ny, sides):
    from hyperflow_gb300 import CartSolver
    from oracle.oracle import Oracle
    case = _case(nx, ny, scheme, sides)
    s, o = CartSolver(case), Oracle(case)
    for n in (1, 2, 10):
        s.run(n)
        o.run(n)
        np.testing.assert_array_equal(s.state(0), o.state(0))
        assert s.time()[:2] == (o.t, o.calls)
    assert s.step() > 0.0
    o.run(1)
    np.testing.assert_array_equal(s.state(0), o.state(0))


def test_paths_mix_and_the_loop_stops_at_the_end_time():
    from hyperflow_gb300 import CartSolver
    a, b = CartSolver(_case(40, 50, "MUSCLHancock", "RTRD", 0.01)), CartSolver(_case(40, 50, "MUSCLHancock", "RTRD", 0.01))
    for n, on in ((3, False), (4, True), (2, False)):
        a.set_block_launches(on)      # True: the fill and a launch per block
        b.set_strict(on)              # True: the fill and one launch for all blocks
        a.run(n)
        b.run(n)
        np.testing.assert_array_equal(a.state(0), b.state(0))
    a.set_block_launches(True)
    assert a.run(1000, clamp_t_end=True) == b.run(1000, clamp_t_end=True) > 0
    assert a.time() == b.time() and a.time()[0] == 0.01
    assert b.run(5, clamp_t_end=True) == 0
    np.testing.assert_array_equal(a.state(0), b.state(0))
