"""What a program may write into the state of a network between runs, on the
dataflow kernel against the path of one launch per tick, bit for bit."""
import numpy as np
import pytest

from tests.test_edge_parity_gpu import DT
from tests.test_flow_gpu import network
from tests.test_gpu_parity import gpu_net

pytestmark = pytest.mark.gpu


def same(nets, names, what):
    for name in names:
        a, b = (net.read(name) for net in nets)
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), f"{what}: {name}"


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("H0", [0, 3])
def test_delays_outside_the_queue_word(variant, H0):
    """bcpnn_set_conn takes delays of 1 to 31 ticks; any other one can be written into di.  A spike sets bit
    di - 1 of the slot's queue word: 32 the sign bit, anything else no bit at all.  Of a source that is published
    and of one that is not (H0), with its spikes before the run set"""
    rng = np.random.default_rng(10 * H0 + variant)
    H, M, C = 6, 20, 90
    pops, projs = network(H, M, C, H0)
    more = {}
    if variant:
        pops = [dict(p, taua=0.05, adgain=1.0) for p in pops]
        more = dict(variant=1, spike_buffer=25)
    nets = [gpu_net(pops, projs, DT, seed=4, poisson_hz=60.0, max_ticks=64, per_tick=p, **more) for p in (False, True)]
    try:
        for q, p in enumerate(projs):
            n = nets[0].info(f"ii_{q}")[1]
            ns = pops[p["src_pop"]]["hcu_num"] * pops[p["src_pop"]]["mcu_num"]
            ii = rng.integers(-1, ns, n).astype(np.int32)
            di = rng.choice(np.array([-32, -1, 0, 1, 2, 5, 31, 32, 33, 63, 64, 2**31 - 1]), n).astype(np.int32)
            si = (rng.random(ns) < 0.5).astype(np.int8)
            for net in nets:
                net.set_conn(q, ii, np.ones(n, np.int32))
                net.write(f"di_{q}", di)
                if not variant or not H0 or p["src_pop"] == 1:
                    net.write(f"si_{q}", si)
        lg = (rng.random(sum(p["hcu_num"] * p["mcu_num"] for p in pops)) * 3 - 3).astype(np.float32)
        t = 1
        for n in (1, 2, 40):
            for net in nets:
                net.set_stimulus(lg, np.ones(sum(p["hcu_num"] for p in pops), np.float32))
                net.run(t, n, 1.0, 1.0)
            t += n
            same(nets, [f"{x}_{q}" for q in range(len(projs))
                        for x in ("qi", ".siq", "di", "pi", "ti", "zi", "pij", "zj2", "wij")] +
                 [f"{x}_{p}" for p in range(len(pops)) for x in ("dsup", "epsc", "bj")], f"after {t - 1} ticks")
        assert nets[0].counters() == nets[1].counters() and nets[0].counters()[0] > 0
    finally:
        for net in nets:
            net.close()
