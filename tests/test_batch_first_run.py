"""A batch's first run, captured by a caller or made in a thread of its own, in the default configuration and
in others selected before it; runs of every length from a few graphs."""
import ctypes as C
import threading

import numpy as np
import pytest


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


@pytest.mark.gpu
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


@pytest.mark.gpu
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


def test_runs_of_all_lengths_come_out_of_24_graphs():
    from test_device_math_host import LIB
    f = C.CDLL(LIB).hm_batch_graph_steps
    f.argtypes, f.restype = [C.c_int64, C.c_int], C.c_int64
    for lengths in ([100] * 5, range(1, 1500), range(300, 0, -1), [100, 7, 2 ** 17 + 5, 100, 1, 999]):
        graphs = set()
        for n in lengths:
            left, pieces = n, 0
            while left > 0:
                k = min(left, 128)
                if k not in graphs:
                    k = f(left, len(graphs))
                assert 1 <= k <= min(left, 128)
                graphs.add(k)
                left -= k
                pieces += 1
            assert pieces <= n // 128 + 7
        assert len(graphs) <= 24
        if len(set(lengths)) == 1:
            assert graphs == set(lengths)      # one graph for a length that repeats


@pytest.mark.gpu
def test_runs_of_many_lengths_equal_one_run():
    a, b = _batches("Godunov", 0)
    lengths = [1, 2, 3, 7, 100, 129, 31, 130, 12, 127, 77, 100, 5, 150, 13, 14, 15, 21, 22, 23, 120, 63, 255]      # past the lengths with a graph of their own
    for n in lengths:
        a.run(n)
    b.run(sum(lengths), graph=False)
    _same(a, b)
    assert a.counters()["steps"] == sum(lengths)
