"""What a step finds of the calls before it: the wave-speed maxima of a TimeStep call or a ghost fill that a
caller's graph ran again, or that no step followed, are not those of the next step's fields; strict mode
switched on after a step was captured stops its replays; a captured TimeStep call is not taken as made."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(n=40):
    from hyperflow_gb300 import CartSolver, cases
    case = cases.quadrant_case(n, scheme="MUSCLHancock", limiter="MinBee", cfl=cases.CFL_2D)
    case["simulation"]["t_end"] = 0.01
    return CartSolver(case)


def _calm(U):
    """The same pressure and density at rest: smaller wave speeds everywhere."""
    U = U.copy()
    U[3] -= 0.5 * (U[1] ** 2 + U[2] ** 2) / U[0]
    U[1:3] = 0.0
    U[3] *= 0.25
    return U


def _next_step(s, U):
    s.set_state(0, U)
    dt = s.step()
    return [dt, s.state(0)]


@pytest.mark.parametrize("path", ["one launch", "fill", "launch per block"])
@pytest.mark.parametrize("call", ["hf_time_step", "hf_apply_bcs"])
def test_a_replayed_call_leaves_no_maxima_to_the_next_step(call, path):
    import torch
    from hyperflow_gb300._lib import lib
    a, b = _solver(), _solver()
    for s in (a, b):
        s.set_strict(path == "fill")               # (strict mode keeps the ghost fill)
        s.set_block_launches(path == "launch per block")
        s.run(12)
    stream = torch.cuda.ExternalStream(a.stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        g.capture_begin(capture_error_mode="thread_local")
        assert (lib().hf_apply_bcs(a._h) if call == "hf_apply_bcs" else lib().hf_time_step(a._h, None)) == 0
        g.capture_end()
        a.step(), b.step()
        for _ in range(2):
            g.replay()
            U = _calm(b.state(0))
            for x, y in zip(_next_step(a, U), _next_step(b, U)):
                np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("path", ["fill", "launch per block"])
def test_a_run_that_has_ended_leaves_no_maxima_to_the_next_step(path):
    """At the end time: a TimeStep call, a clamped run that takes no step, then calmer fields."""
    a, b = _solver(), _solver()
    for s in (a, b):
        s.set_strict(path == "fill")
        s.set_block_launches(path == "launch per block")
        assert s.run(1000, clamp_t_end=True) > 5 and s.time()[0] == 0.01
    a.calculate_time_step()
    assert a.run(3, clamp_t_end=True) == 0
    U = _calm(b.state(0))
    for x, y in zip(_next_step(a, U), _next_step(b, U)):
        np.testing.assert_array_equal(x, y)


def test_strict_mode_stops_steps_captured_before_it():
    import torch
    from hyperflow_gb300 import CartSolver, HyperFlowError, cases
    from hyperflow_gb300._lib import lib
    case = cases.shock_bubble_case(128, cfl=0.8)
    a, b = CartSolver(case), CartSolver(case)
    a.step(), b.step()
    stream = torch.cuda.ExternalStream(a.stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        g.capture_begin(capture_error_mode="thread_local")
        assert lib().hf_step(a._h, None) == 0
        g.capture_end()
        a.set_strict(True)
        for _ in range(100):
            g.replay()
    b.set_strict(True)
    with pytest.raises(HyperFlowError, match="step 82"):
        b.run(100, graph=False)
    with pytest.raises(HyperFlowError, match="step 82"):
        a.sync()
    assert a.time() == b.time()
    np.testing.assert_array_equal(a.state(0), b.state(0))
    assert a.last_nonpositive_cell() == b.last_nonpositive_cell()


@pytest.mark.parametrize("scheme", ["Godunov", "MUSCLHancock"])
@pytest.mark.parametrize("call", ["hf_time_step", "hf_apply_bcs"])
def test_a_call_that_was_only_captured_is_not_taken_as_made(call, scheme):
    """hf_advance after it starts the step itself, and the step after that finds its own wave speeds."""
    import torch
    from hyperflow_gb300 import CartSolver, cases
    from hyperflow_gb300._lib import lib
    case = cases.quadrant_case(40, scheme=scheme, limiter="VanLeer" if scheme == "MUSCLHancock" else None, cfl=cases.CFL_2D)
    case["mesh"]["blocks"][0]["boundaries"]["left"] = {"type": "Dirichlet", "variables": "Primitive",
                                                       "flow_state": [0.5, 9.0, 0.3, 4.0]}
    a, b = CartSolver(case), CartSolver(case)
    for s in (a, b):
        s.run(12)
    stream = torch.cuda.ExternalStream(a.stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        g.capture_begin(capture_error_mode="thread_local")
        assert (lib().hf_apply_bcs(a._h) if call == "hf_apply_bcs" else lib().hf_time_step(a._h, None)) == 0
        g.capture_end()
    for s in (a, b):
        s.advance(1e-3)
    np.testing.assert_array_equal(a.state(0), b.state(0))
    assert a.calculate_time_step() == b.calculate_time_step()
    # captured together, the TimeStep call serves the advance behind it
    h = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        h.capture_begin(capture_error_mode="thread_local")
        assert lib().hf_apply_bcs(a._h) == 0 and lib().hf_time_step(a._h, None) == 0
        a.advance(2e-4)
        h.capture_end()
        h.replay()
        h.replay()
    for _ in range(2):
        b.apply_bcs()
        b.calculate_time_step()
        b.advance(2e-4)
    np.testing.assert_array_equal(a.state(0), b.state(0))
    assert a.time() == b.time()


def test_fields_uploaded_after_a_ghost_fill_have_their_own_predictor():
    a, b = _solver(), _solver()
    U = None
    for s in (a, b):
        s.run(12)
        U = _calm(s.state(0)) if U is None else U
        if s is a:
            s.apply_bcs()
        s.set_state(0, U)
        s.advance(1e-3)
    np.testing.assert_array_equal(a.state(0), b.state(0))
    assert a.calculate_time_step() == b.calculate_time_step()
