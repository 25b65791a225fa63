"""A batch's first run, captured by a caller or made in a thread of its own, in the default configuration and
in others selected before it."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batches(scheme, config, count=2):
    from hyperflow_gb300 import BatchSolver, cases
    spec = {"cases": [cases.quadrant_case(n, scheme=scheme, limiter="MinBee" if scheme != "Godunov" else None,
                                          cfl=cases.CFL_2D) for n in (20, 33)]}
    out = [BatchSolver(spec) for _ in range(count)]
    for b in out:
        if config:
            b.set_config(config)
    return out


def _same(a, b):
    a.sync()
    b.sync()
    for i in range(2):
        np.testing.assert_array_equal(a.state(i), b.state(i))
        assert a.instance_time(i) == b.instance_time(i)


@pytest.mark.parametrize("scheme", ["Godunov", "MUSCLHancock"])
@pytest.mark.parametrize("config", [0, 1, 4])
def test_a_first_run_may_be_captured(scheme, config):
    import torch
    a, b = _batches(scheme, config)
    stream = torch.cuda.ExternalStream(a.stream())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        g.capture_begin(capture_error_mode="thread_local")
        a.run(3, graph=False)
        g.capture_end()
        g.replay()
        g.replay()
    b.run(6)
    _same(a, b)


@pytest.mark.parametrize("config", [0, 3])
def test_a_first_run_in_another_thread(config):
    a, b = _batches("MUSCLHancock", config)
    failed = []

    def work():
        try:
            a.run(4)
        except Exception as e:
            failed.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not failed
    b.run(4)
    _same(a, b)
