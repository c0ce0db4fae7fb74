"""Errors in the dataflow kernel, without a fault: a wait that runs out on a
spike word that nothing publishes, and a slot whose source does not exist.
Either is reported, and after a reset the network runs as a new one does."""
import time

import numpy as np
import pytest

from gsbn_b200 import capi
from tests.test_edge_parity_gpu import DT
from tests.test_flow_gpu import pop, proj
from tests.test_flow_state_gpu import same
from tests.test_gpu_parity import gpu_net

pytestmark = pytest.mark.gpu

STATE = ("dsup_0", "epsc_0", "bj_0", "wij_0", "qi_0", ".siq_0")


def pair(H, M, C, variant):
    pops, more = [pop(H, M)], {}
    if variant:
        pops, more = [dict(pops[0], taua=0.05, adgain=1.0)], dict(variant=1, spike_buffer=25)
    nets = [gpu_net(pops, [proj(0, 0, C)], DT, seed=4, poisson_hz=40.0, max_ticks=64, per_tick=p, **more)
            for p in (False, True)]
    rng = np.random.default_rng(H)
    ii, di = rng.integers(-1, H * M, H * C).astype(np.int32), rng.integers(1, 4, H * C).astype(np.int32)
    for net in nets:
        net.set_conn(0, ii, di)
        net.set_stimulus(np.zeros(H * M, np.float32), np.ones(H, np.float32))
    return nets, ii, di


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("H,M,C", [(1, 5, 5), (9, 40, 70), (160, 33, 40)])
def test_a_wait_that_runs_out(H, M, C, variant):
    nets, _, _ = pair(H, M, C, variant)
    try:
        nets[0].run(1, 30, 1.0, 1.0)
        nets[0].sync()
        t0 = time.perf_counter()
        rc, msg = nets[0].selftest_flow_timeout(20_000_000)
        assert 0.015 < time.perf_counter() - t0 < 5.0
        assert rc == -6 and "timed out" in msg, msg
        nets[0].sync()  # the error was reported once
        nets[0].reset()
        for net in nets:
            for first, n in ((1, 20), (21, 3)):
                net.run(first, n, 1.0, 1.0)
        assert np.array_equal(nets[0].spike_log(0), nets[1].spike_log(0))
        same(nets, STATE, "after the reset")
        assert nets[0].selftest_flow_timeout(10)[0] == -1   # limit out of range
        assert nets[1].selftest_flow_timeout(10**6)[0] == -5  # one launch per tick
    finally:
        for net in nets:
            net.close()


@pytest.mark.parametrize("variant", [0, 1])
def test_a_source_that_does_not_exist(variant):
    """written into ii (bcpnn_set_conn refuses it): the slot is left out, the run goes on to its end as in the
    per-tick path, and the error is reported"""
    H, M, C = 60, 20, 50
    nets, ii, di = pair(H, M, C, variant)
    try:
        bad = ii.copy()
        bad[7 * C + 3] = H * M
        for net in nets:
            net.write("ii_0", bad)
            net.run(1, 50, 1.0, 1.0)
        same(nets, STATE, "with the error")
        for net in nets:
            with pytest.raises(capi.BcpnnError, match="outside the source population"):
                net.sync()
            net.set_conn(0, ii, di)
            net.reset()
            net.run(1, 50, 1.0, 1.0)
            net.sync()
        same(nets, STATE, "after the reset")
    finally:
        for net in nets:
            net.close()
