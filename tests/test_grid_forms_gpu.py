"""The CTA size that the plain path takes by default, by the number of HCUs: 512
threads while the grid of one CTA per HCU is resident at once, then 256, then
128, else one launch per tick.  At the sizes where the choice changes, and
with columns of more than one work unit and of many cells per thread: spikes,
state and counters bit-identical to the oracle, and the launches of a run."""
import numpy as np
import pytest

from gsbn_b200 import capi
from oracle import sim
from tests.harness import first_mismatch, state
from tests.test_edge_parity_gpu import DT, runs_of
from tests.test_gpu_parity import spikes_of

pytestmark = pytest.mark.gpu

# HCUs, MCUs, slots per HCU; whether a run is one launch on a GPU of 148 SMs
CASES = [(148, 5, 40, True), (149, 5, 40, True), (296, 7, 300, True), (297, 7, 300, True), (300, 20, 517, True),
         (297, 100, 60, True), (592, 3, 20, True), (593, 3, 20, False), (149, 257, 20, False), (297, 129, 20, False)]


@pytest.mark.parametrize("H,M,C,one_launch", CASES)
def test_default_form(H, M, C, one_launch):
    rng = np.random.default_rng(H + M)
    pops = [dict(hcu_num=H, mcu_num=M, taum=0.005, wtagain=1.0, maxfq=400.0, igain=1.0, wgain=1.0, lgbias=0.0, snoise=0.0)]
    projs = [dict(src_pop=0, dest_pop=0, tauzi=0.01, tauzj=0.012, taue=0.02, taup=1.0, maxfq=400.0, bgain=1.0, wgain=1.0,
                  tauepsc=0.0, slot_num=float(C))]
    ii = np.concatenate([np.sort(rng.choice(H * M, C, replace=False)) for _ in range(H)]).astype(np.int32)
    di = rng.integers(1, 4, H * C).astype(np.int32)
    orc = sim.OracleNet(pops, projs, DT, seed=9)
    gpu = capi.Net(pops, projs, DT, seed=9, max_ticks=64)
    try:
        orc.set_conn(0, ii, di)
        gpu.set_conn(0, ii, di)
        for first, n, prn, old_prn, lg, wm in runs_of(pops, rng, n_train=2, n_recall=1, train=20, recall=15):
            orc.set_stimulus(lg, wm)
            gpu.set_stimulus(lg, wm)
            want = orc.run(first, n, prn, old_prn)
            before = gpu.kernel_launches()
            gpu.run(first, n, prn, old_prn)
            launches = gpu.kernel_launches() - before
            assert (launches < n) == one_launch, launches
            got = spikes_of(gpu, pops, n)
            for t in range(n):
                assert np.array_equal(want[t][0], got[t][0]), f"spikes differ at simstep {first + t}"
        msg = first_mismatch(state(orc, 1, 1), state(gpu, 1, 1))
        assert msg is None, msg
        assert orc.counters() == gpu.counters()
    finally:
        gpu.close()
