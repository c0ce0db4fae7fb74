"""Which kernel the parity tests' networks run on: the cases that are meant for
the dataflow kernel take it, and the others do not.  (A parity test alone
passes on any kernel.)  Sizes are for a GPU of 148 SMs."""
import numpy as np
import pytest

from tests import test_flow_gpu, test_flow_multi_gpu, test_grid_forms_gpu, test_recall_events_gpu
from tests.test_edge_parity_gpu import DT
from tests.test_flow_gpu import network, pop, proj
from tests.test_gpu_parity import gpu_net

pytestmark = pytest.mark.gpu


def cases(test):
    """the parameter sets of a parametrised test"""
    marks = [m for m in test.pytestmark if m.name == "parametrize"]
    assert len(marks) == 1
    return marks[0].args[1]


def form(pops, projs, **kw):
    net = gpu_net(pops, projs, DT, seed=1, max_ticks=8, **kw)
    try:
        return net.run_form()
    finally:
        net.close()


@pytest.mark.parametrize("H,M,C,H0", cases(test_flow_gpu.test_against_per_tick))
def test_lazy(H, M, C, H0):
    pops, projs = network(H, M, C, H0)
    assert form(pops, projs) == ("dataflow" if M <= 128 else "barrier", 512 if H + H0 <= 148 else 256)
    assert form(pops, projs, per_tick=True)[0] == "per tick"


@pytest.mark.parametrize("H,M,C,H0,ring,flow", cases(test_flow_multi_gpu.test_against_per_tick))
def test_multi(H, M, C, H0, ring, flow):
    pops, projs = network(H, M, C, H0)
    pops = [dict(p, taua=0.05, adgain=1.0) for p in pops]
    kw = dict(variant=1, spike_buffer=ring)
    assert form(pops, projs, **kw)[0] == ("dataflow" if flow else "barrier")
    assert form(pops, projs, per_tick=True, **kw)[0] == "per tick"
    assert form(pops, projs, per_tick="global", **kw)[0] == ("barrier" if H <= 148 else "per tick")


@pytest.mark.parametrize("H,M,C,one_launch", test_grid_forms_gpu.CASES)
def test_default_by_hcus(H, M, C, one_launch):
    want = ("dataflow", 512 if H <= 148 else 256) if H <= 296 and M <= 128 else \
        ("barrier", 128) if one_launch else ("per tick", 512)
    assert form([pop(H, M)], [proj(0, 0, C)]) == want


def test_external_spikes_leave_the_dataflow_kernel():
    for kw, threads in ((dict(), 512), (dict(tick_threads=256), 256), (dict(fp64_tables=1), 512)):
        net = gpu_net([pop(8, 32)], [proj(0, 0, 64)], DT, seed=1, max_ticks=8, **kw)
        assert net.run_form() == ("dataflow", threads)
        net.set_ext_spikes(0, {1: [3]})
        assert net.run_form() == ("barrier", threads)
        net.close()


@pytest.mark.parametrize("H,M,R,hz,events", [(*c, c[3] < 200.0) for c in cases(test_recall_events_gpu.test_epsc_bits)])
def test_recall_contraction(H, M, R, hz, events):
    """by events: a launch more per tick, for the spike lists"""
    rng = np.random.default_rng(1)
    W = np.zeros((H * M, H * M), np.float32)
    for value, launches in ((0.0, 3 if events else 2), (np.inf, 2)):
        W[0, 0] = value
        _, eng = test_recall_events_gpu.engine(H, M, R, hz, rng, W)
        before = eng.launches()
        eng.run(10, 4)
        assert eng.launches() - before == 4 * launches
        eng.close()
