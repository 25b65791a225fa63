"""The dt and step count a step leaves in host memory: steps, host-buffer steps, device loops (clamped
ones too), single calls, restores and captured steps in turn, against the path of a launch per block, which
copies dt from the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pinned(a):
    import torch
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _host_step(s, nb):
    ins = [_pinned(s.state(b)) for b in range(nb)]
    outs = [_pinned(u) for u in ins]
    dt = s.step_io(ins, outs)
    return [dt, *outs]


@pytest.mark.parametrize("kind", ["one tile", "one block", "three blocks"])
def test_results_in_host_memory_follow_every_way_of_stepping(kind):
    from hyperflow_gb300 import CartSolver, cases
    if kind == "three blocks":
        case = cases.forward_facing_step_case(30, limiter="MinBee")
    else:
        n = 12 if kind == "one tile" else 90
        case = cases.quadrant_case(n, scheme="MUSCLHancock", limiter="VanLeer", cfl=cases.CFL_2D)
    case["simulation"]["t_end"] = 1.0e9
    a, b = CartSolver(case), CartSolver(case)
    b.set_block_launches(True)
    nb = len(case["mesh"]["blocks"])
    blob = [s.checkpoint() for s in (a, b)]
    moves = [lambda s: [s.step()], lambda s: _host_step(s, nb), lambda s: [s.run(3)],
             lambda s: [s.run(2, clamp_t_end=True)], lambda s: [s.step(), s.step()], lambda s: _host_step(s, nb),
             lambda s: [s.apply_bcs(), s.advance(s.calculate_time_step())], lambda s: _host_step(s, nb),
             lambda s: [s.run(1, graph=False)], lambda s: [s.step()]]
    for k, move in enumerate(moves + moves):
        if k == len(moves):
            a.restore(blob[0])
            b.restore(blob[1])
        got, ref = move(a), move(b)
        for x, y in zip(got, ref):
            np.testing.assert_array_equal(x, y)
        for i in range(nb):
            np.testing.assert_array_equal(a.state(i), b.state(i))
        assert a.time() == b.time()


def test_a_captured_step_holds_all_of_itself():
    import torch
    from hyperflow_gb300 import CartSolver, cases
    from hyperflow_gb300._lib import lib
    case = cases.quadrant_case(48, scheme="MUSCLHancock", limiter="MinBee", cfl=cases.CFL_2D)
    case["simulation"]["t_end"] = 1.0e9
    a, b = CartSolver(case), CartSolver(case)
    a.step(), b.step()
    stream = torch.cuda.ExternalStream(a.stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        g.capture_begin(capture_error_mode="thread_local")
        assert lib().hf_step(a._h, None) == 0
        g.capture_end()
        a.run(2, clamp_t_end=True)     # the loop's clamp switch stays on behind it
        g.replay()
        U = a.state(0)
        a.set_state(0, U[:, ::-1].copy())
        g.replay()
        a.run(1, clamp_t_end=True)
        assert a.run(1, clamp_t_end=True) == 1
        g.replay()
        out = _host_step(a, 1)
    b.run(3)
    b.set_state(0, b.state(0)[:, ::-1].copy())
    b.run(4)
    ref = _host_step(b, 1)
    assert out[0] == ref[0]
    np.testing.assert_array_equal(out[1], ref[1])
    np.testing.assert_array_equal(a.state(0), b.state(0))
    assert a.time() == b.time()


@pytest.mark.parametrize("edge", [False, True])
def test_unstructured_loops_of_many_steps_a_graph(edge):
    """Runs past a graph's 32 steps, clamped ones that stop inside one, and mode changes between them."""
    from hyperflow_gb300 import UnsSolver, meshgen
    from test_uns import load
    g = load("tri_hole_3k")
    case, text = g["case"], meshgen.hmsh_text(g["verts"], g["codes"])
    first = UnsSolver(case, mesh_text=text)
    first.run(70)
    case["simulation"]["t_end"] = 1.6 * first.time()[0]
    a, b = UnsSolver(case, mesh_text=text), UnsSolver(case, mesh_text=text)
    for s in (a, b):
        s.set_edge_mode(edge)
    a.run(70)
    b.run(70, graph=False)
    np.testing.assert_array_equal(a.state(), b.state())
    for s in (a, b):
        s.set_edge_mode(not edge)
    assert a.run(1000, clamp_t_end=True) == b.run(1000, clamp_t_end=True, graph=False) > 0
    assert a.time() == b.time() and a.time()[0] == case["simulation"]["t_end"]
    np.testing.assert_array_equal(a.state(), b.state())
    assert a.run(40, clamp_t_end=True) == 0


def test_a_strict_stop_leaves_the_count_to_the_device():
    """In strict mode a step that does not run, for a failure recorded before it, leaves no result; the
    host-buffer step after it still finds the right buffers."""
    from hyperflow_gb300 import CartSolver, HyperFlowError, cases
    case = cases.shock_bubble_case(128, cfl=0.8)
    a, b = CartSolver(case), CartSolver(case)
    for s in (a, b):
        s.step()
        s.set_strict(True)
        with pytest.raises(HyperFlowError, match="step 82"):
            s.run(200)
        with pytest.raises(HyperFlowError, match="step 82"):
            s.step()
        s.set_strict(False)
        s.clear_error_cell()
        b.set_block_launches(True)
    assert a.time() == b.time()
    got, ref = _host_step(a, 1), _host_step(b, 1)
    assert got[0] == ref[0]
    np.testing.assert_array_equal(got[1], ref[1])


@pytest.mark.parametrize("scheme", ["Godunov", "MUSCLHancock"])
def test_a_batch_run_may_be_captured(scheme):
    import torch
    from hyperflow_gb300 import BatchSolver, cases
    spec = {"cases": [cases.quadrant_case(n, scheme=scheme, limiter="MinBee" if scheme != "Godunov" else None,
                                          cfl=cases.CFL_2D) for n in (20, 33)]}
    a, b = BatchSolver(spec), BatchSolver(spec)
    if scheme != "Godunov":      # (its tensor maps are made by the first run)
        a.run(1, graph=False), b.run(1, graph=False)
    a.sync()
    stream = torch.cuda.ExternalStream(a.stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        g.capture_begin(capture_error_mode="thread_local")
        a.run(3, graph=False)
        g.capture_end()
        g.replay()
        g.replay()
    a.sync()
    b.run(6)
    b.sync()
    for i in range(2):
        np.testing.assert_array_equal(a.state(i), b.state(i))
