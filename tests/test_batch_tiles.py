"""Batched cases with a tile shape per case: sides below, at and past the tiles' edges, runs longer
than one graph, and the upload of one case, against the oracle run on each case alone, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDES = [4, 5, 17, 33, 64, 65, 131]


def _oracle(case, steps, width):
    from oracle.oracle import Oracle
    o = Oracle(case, nthreads=4)
    o.run(steps)
    return o.state(0)[:, width:-width, width:-width], o.t


@pytest.mark.parametrize("scheme,limiter", [("Godunov", None), ("MUSCLHancock", "MinBee"), ("MUSCLHancock", "VanLeer")])
@pytest.mark.parametrize("config", [0, 1])
def test_case_tiles_match_the_oracle(port_lib, scheme, limiter, config):
    from hyperflow_gb300 import BatchSolver, cases
    specs = [cases.quadrant_case(n, scheme=scheme, limiter=limiter, cfl=cases.CFL_2D) for n in SIDES]
    width = 1 if scheme == "Godunov" else 2
    steps = 130 if config == 0 and limiter != "VanLeer" else 14   # past one graph's 128 steps
    b = BatchSolver({"cases": specs})
    b.set_config(config)
    b.run(steps, graph=config == 0)
    b.sync()
    for i, c in enumerate(specs):
        ref, t = _oracle(c, steps, width)
        np.testing.assert_array_equal(b.state(i), ref, err_msg=f"side {SIDES[i]}")
        assert b.instance_time(i)[0] == t
    assert b.counters()["steps"] == steps


def test_upload_of_one_case_leaves_the_others(port_lib):
    from hyperflow_gb300 import BatchSolver, cases
    specs = [cases.quadrant_case(n, scheme="MUSCLHancock", limiter="MinBee", cfl=cases.CFL_2D) for n in (40, 51, 64)]
    a, b = BatchSolver({"cases": specs}), BatchSolver({"cases": specs})
    a.run(12), b.run(12)
    for i in range(3):
        U = a.state(i)
        if i == 1:
            U = U[:, ::-1, ::-1].copy()
            U[1:3] *= -0.5
            U[3] *= 1.5
            a.set_state(1, U)
        b.set_state(i, U)      # every case uploaded again: all maxima formed anew
    a.run(9), b.run(9)
    for i in range(3):
        np.testing.assert_array_equal(a.state(i), b.state(i))
        assert a.instance_time(i) == b.instance_time(i)
