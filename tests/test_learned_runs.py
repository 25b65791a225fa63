"""Learned runs in many calls: of one step, of odd and even numbers of steps, of none, plain and with the
network in turn, with the settings changed between them, against the same steps one by one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pair(n):
    from oracle import mlp_oracle as M
    from hyperflow_gb300 import CartSolver, cases
    from hyperflow_gb300.learned import LearnedSolver, init_params
    s = CartSolver(cases.shock_bubble_case(n))
    s.run(5)
    U0 = s.state(0)[:, 2:-2, 2:-2].astype(np.float32)
    s.close()
    p = init_params(3, out_scale=0.05)
    p[M.OFF_B3:] = [0.05, -0.03, 0.04, -0.2]
    out = []
    for _ in range(2):
        L = LearnedSolver(n, 1.0 / n)
        L.set_params(p)
        L.set_state(U0)
        out.append(L)
    return out


@pytest.mark.parametrize("fused", [0, 1, 2])
def test_runs_in_many_calls_equal_single_steps(fused):
    a, b = _pair(48)
    for L in (a, b):
        L.set_fused(fused)
    t, steps = 0.0, 0
    # per call: how many of the current dt it goes on for, with the network or plain, what is set before it
    calls = [(0.6, 1, None), (2.5, 1, None), (0.0, 1, None), (-1.0, 0, None), (0.5, 0, None), (3.4, 1, None),
             (4.6, 1, None), (1.5, 0, None), (6.3, 1, None), (7.2, 0, None), (0.4, 1, 1), (5.5, 1, None), (5.5, 0, None),
             (4.5, 1, 0), (4.5, 1, None), (70.5, 1, None), (9.5, 0, None), (1.0, 1, None), (2.0, 1, None)]
    rejected = 0
    for span, mlp, guard in calls:
        for L in (a, b):
            if guard is not None:
                L.set_guard_mode(guard)
        t_end = t + span * (b.cfl_dt() * (0.2 if steps < 5 else 1.0))
        k = rej = 0
        while t < t_end:
            dt = b.cfl_dt() * (0.2 if steps < 5 else 1.0)
            if t + dt > t_end:
                dt = t_end - t
            rej += b.step(dt, bool(mlp))
            t += dt
            steps += 1
            k += 1
        assert a.run_to(t_end, bool(mlp)) == (k, rej)
        np.testing.assert_array_equal(a.state().view(np.uint32), b.state().view(np.uint32))
        rejected += rej
    assert steps > 100 and rejected > 0
    a.close()
    b.close()
