"""A batch run's spike logs: they hold the spikes of that run alone, whatever
ran before and however many ticks the engine has room for, and what a run costs
depends on its ticks, not on that room."""
import statistics

import numpy as np
import pytest
import torch

from gsbn_b200 import batch

pytestmark = pytest.mark.gpu


def engine(shapes, max_ticks):
    ms = [batch.make_members(n=1, seed=50 + k, hcu=(H, H), mcu=(M, M), n_patterns=2)[0] for k, (H, M) in enumerate(shapes)]
    return batch.BatchEngine(ms, max_ticks=max_ticks)


def test_logs_of_runs_of_many_lengths():
    """a log of 64 x 50 MCUs over 64 ticks is of several parts, one of 8 x 5 of one in part"""
    shapes = [(8, 5), (64, 50), (20, 12)]
    engs = [engine(shapes, m) for m in (64, 5000)]
    try:
        t, total = 1, 0
        for n in (64, 5, 1, 33, 64, 2):
            for eng in engs:
                eng.run_segment(t, n, 1.0, 1.0, 0, 0)
            t += n
            for m in range(len(shapes)):
                a, b = (eng.spike_log(m) for eng in engs)
                assert a.shape[0] == n and np.array_equal(a, b)
                total += int(np.unpackbits(a.view(np.uint8)).sum())
        # every spike is in one run's log: the logs' bits are the counters of spikes since the start
        counted = sum(int(engs[0].read(m, ".counter_0").sum()) for m in range(len(shapes)))
        assert total == counted > 0
    finally:
        for eng in engs:
            eng.close()


def test_cost_of_room():
    """2^21 ticks of 64 x 50 MCUs are 839 MB, which no B200 writes in less than 100 us"""
    us = []
    for max_ticks in (128, 1 << 21):
        eng = engine([(64, 50)], max_ticks)
        stream = torch.cuda.ExternalStream(eng.stream())
        times = []
        for k in range(30):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record(stream)
            eng.run_segment(1 + k, 1, 1.0, 1.0, 0, 0)
            b.record(stream)
            eng.sync()
            times.append(a.elapsed_time(b) * 1e3)
        us.append(statistics.median(times[5:]))
        eng.close()
    print("us per run of one tick:", us)
    assert us[1] < us[0] + 50, us
