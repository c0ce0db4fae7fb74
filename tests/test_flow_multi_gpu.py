"""ProcUpdMulti on the dataflow kernel where it can go wrong: MCU counts at the
warps of the population update and one beyond the kernel's range, HCU counts at
each CTA size, rings of 1, 25 and 32 ticks and one beyond its masks, odd slot
counts and empty slots, several projections, runs of 1 to 6 ticks, and spikes
and queue words written before a run.  Bit-identical to the path of one launch
per tick; two populations of which one is never published take the other one."""
import numpy as np
import pytest

from tests.harness import STATE_POP
from tests.test_edge_parity_gpu import DT
from tests.test_flow_gpu import RUNS, network
from tests.test_gpu_parity import gpu_net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,M,C,H0,ring,flow", [
    (3, 1, 3, 0, 25, True), (16, 31, 77, 0, 32, True), (8, 33, 129, 0, 1, True), (5, 64, 320, 0, 2, True),
    (6, 65, 131, 0, 25, True), (4, 128, 511, 0, 25, True), (150, 9, 41, 0, 25, True), (150, 100, 37, 0, 7, True),
    (4, 129, 100, 0, 25, False), (8, 32, 256, 0, 33, False), (8, 33, 129, 3, 25, False)])
def test_against_per_tick(H, M, C, H0, ring, flow):
    rng = np.random.default_rng(H * 1000 + M + ring)
    pops, projs = network(H, M, C, H0)
    if H <= 16 and not H0:
        projs = projs + [dict(projs[0], slot_num=float(max(1, C // 2)), tauzi=0.005)]
    pops = [dict(p, taua=0.05, adgain=1.0) for p in pops]
    nets = [gpu_net(pops, projs, DT, seed=4, poisson_hz=40.0, max_ticks=64, per_tick=p, variant=1, spike_buffer=ring)
            for p in (False, True)]
    try:
        for q, p in enumerate(projs):
            ns = pops[p["src_pop"]]["hcu_num"] * pops[p["src_pop"]]["mcu_num"]
            Hd, Cq = pops[p["dest_pop"]]["hcu_num"], min(ns, int(p["slot_num"]))
            ii = np.concatenate([rng.choice(ns, Cq, replace=False) for _ in range(Hd)]).astype(np.int32)
            ii[rng.random(ii.size) < 0.1] = -1
            di = rng.integers(1, 32 if q == 1 else 4, ii.size).astype(np.int32)
            for net in nets:
                net.set_conn(q, ii, di)
        t, prn, launches = 1, 0.0, [net.kernel_launches() for net in nets]
        lg = (rng.random(sum(p["hcu_num"] * p["mcu_num"] for p in pops)) * 3 - 3).astype(np.float32)
        wm = np.ones(sum(p["hcu_num"] for p in pops), np.float32)
        for k, n in enumerate(RUNS):
            now = 0.0 if k in (4, 8) else 1.0
            if k in (2, 5, 8):
                for q in range(len(projs)):
                    si = (rng.random(nets[0].info(f"si_{q}")[1]) < 0.3).astype(np.int8)
                    qi = (rng.integers(0, 2**31, nets[0].info(f"qi_{q}")[1]) & rng.integers(0, 2**31) & 0x11111111)
                    for net in nets:
                        if not H0 or projs[q]["src_pop"] == 1:  # of a published population
                            net.write(f"si_{q}", si)
                        net.write(f"qi_{q}", qi.astype(np.int32))
            logs = []
            for net in nets:
                net.set_stimulus(lg, wm)
                net.run(t, n, now, prn)
                logs.append([net.spike_log(p) for p in range(len(pops))] + [net.ss_flags()])
            for p, (a, b) in enumerate(zip(*logs)):
                assert np.array_equal(a, b), f"run {k}: log {p}"
            names = [f"{x}_{p}" for p in range(len(pops)) for x in (*STATE_POP, "ada", "spike")]
            names += [f"{x}_{q}" for q in range(len(projs))
                      for x in ("pi", "ei", "zi", "ti", "pj", "ej", "zj", "pij", "eij", "zj2", "wij", "qi", "si", ".siq")]
            for name in names:
                a, b = (net.read(name) for net in nets)
                assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), f"run {k}: {name}"
            t, prn = t + n, now
        assert nets[0].counters() == nets[1].counters()
        assert sum(nets[0].counters()) > 0
        if flow:
            assert nets[0].kernel_launches() - launches[0] < nets[1].kernel_launches() - launches[1]
    finally:
        for net in nets:
            net.close()
