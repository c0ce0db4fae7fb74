"""ProcUpdMulti over runs that skip ticks or repeat them, against the compiled
restatement: a row that was written with a later tick decays over a negative
number of ticks (gsbn's expressions, ProcUpdMulti/Proj.cpp:409-488, without a
test), which no table holds.  On every form of the launch, with the ring walked
(40 ticks, and one launch per tick) and as a mask."""
import numpy as np
import pytest

from oracle import multi
from tests.test_edge_parity_gpu import DT
from tests.test_flow_gpu import pop, proj
from tests.test_gpu_parity import gpu_net
from tests.test_multi_gpu import ARRAYS

pytestmark = pytest.mark.gpu

RUNS = ((1, 6, 1.0), (9, 5, 1.0), (60, 4, 1.0), (61, 5, 1.0), (63, 2, 1.0), (30, 8, 1.0), (38, 1, 0.0), (39, 3, 0.0),
        (20, 3, 0.0), (400, 5, 1.0), (405, 6, 1.0), (1, 3, 1.0))


@pytest.mark.parametrize("ring,per_tick", [(25, False), (25, True), (25, "global"), (40, False), (3, True), (32, False)])
def test_against_the_restatement(ring, per_tick):
    rng = np.random.default_rng(ring)
    H, M, C = 6, 31, 80
    pops = [dict(pop(H, M), snoise=0.0, taua=0.05, adgain=1.0)]
    projs = [proj(0, 0, C)]
    gpu = gpu_net(pops, projs, DT, seed=4, max_ticks=64, variant=1, spike_buffer=ring, per_tick=per_tick)
    orc = multi.MultiNetC(pops, projs, DT, seed=4, spike_buffer=ring)
    ii, di = rng.integers(-1, H * M, H * C).astype(np.int32), rng.integers(1, 6, H * C).astype(np.int32)
    lg = (rng.random(H * M) * 3 - 3).astype(np.float32)
    try:
        for net in (gpu, orc):
            net.set_conn(0, ii, di)
            net.set_stimulus(lg, np.ones(H, np.float32))
        old, spikes = 0.0, 0
        for first, n, prn in RUNS:
            gpu.run(first, n, prn, old)
            want = orc.run(first, n, prn, old)
            old = prn
            got = gpu.spike_log(0)
            assert np.array_equal(got, want[0]), f"spikes from {first}"
            spikes += int(np.unpackbits(got.view(np.uint8)).sum())
            for name in ARRAYS:
                a = gpu.read(name)
                b = np.asarray(orc.read(name)).astype(a.dtype)
                # weights of a trace that such a decay makes negative are NaN, of which the bits are not defined
                same = a.view(np.uint8 if a.itemsize == 1 else np.uint32) == b.view(np.uint8 if b.itemsize == 1 else np.uint32)
                assert np.all(same | (np.isnan(a) & np.isnan(b))), f"{name} from {first}"
        assert spikes > 50
    finally:
        gpu.close()
