"""The dataflow kernel of the plain path where it can go wrong: MCU counts at
the warps of the population update and one beyond the kernel's range, HCU
counts at each CTA size, odd slot counts, runs of 1 to 6 ticks (its events and
spike words are kept for a few ticks), spikes written into the state before a
run for projections whose source is published and for one whose is not, and
empty slots.  Bit-identical to the path of one launch per tick."""
import numpy as np
import pytest

from tests.harness import STATE_POP
from tests.test_edge_parity_gpu import DT, runs_of
from tests.test_gpu_parity import gpu_net

pytestmark = pytest.mark.gpu

RUNS = (1, 2, 3, 4, 5, 6, 2, 1, 33, 2)


def pop(H, M):
    return dict(hcu_num=H, mcu_num=M, taum=0.005, wtagain=1.0, maxfq=500.0, igain=1.0, wgain=1.0, lgbias=0.0, snoise=0.1)


def proj(src, dest, C, tauzi=0.01):
    return dict(src_pop=src, dest_pop=dest, tauzi=tauzi, tauzj=0.012, taue=0.02, taup=1.0, maxfq=500.0, bgain=1.0,
                wgain=1.0, tauepsc=0.0, slot_num=float(C))


def network(H, M, C, H0):
    """population 0 (H0 HCUs, not the destination of any projection: never published) -> 1, and 1 -> 1 twice"""
    pops, projs = [pop(H, M)], [proj(0, 0, C)]
    if H0:
        pops = [pop(H0, 5), pop(H, M)]
        projs = [proj(0, 1, 5 * H0), proj(1, 1, C), proj(1, 1, max(1, C // 2), 0.005)]
    return pops, projs


@pytest.mark.parametrize("H,M,C,H0", [(3, 1, 3, 0), (16, 31, 77, 4), (8, 32, 256, 3), (8, 33, 129, 3), (5, 64, 320, 0),
                                      (6, 65, 131, 2), (4, 128, 511, 2), (4, 129, 100, 2), (150, 9, 41, 0),
                                      (150, 33, 65, 0), (150, 100, 37, 3)])
def test_against_per_tick(H, M, C, H0):
    rng = np.random.default_rng(H * 1000 + M)
    pops, projs = network(H, M, C, H0)
    nets = [gpu_net(pops, projs, DT, seed=4, poisson_hz=15.0, max_ticks=64, per_tick=p) for p in (False, True)]
    try:
        for q, p in enumerate(projs):
            ns = pops[p["src_pop"]]["hcu_num"] * pops[p["src_pop"]]["mcu_num"]
            Hd, Cq = pops[p["dest_pop"]]["hcu_num"], min(ns, int(p["slot_num"]))
            ii = np.concatenate([rng.choice(ns, Cq, replace=False) for _ in range(Hd)]).astype(np.int32)
            ii[rng.random(ii.size) < 0.1] = -1
            di = rng.integers(1, 32 if q == 1 else 4, ii.size).astype(np.int32)
            for net in nets:
                net.set_conn(q, ii, di)
        t, prn = 1, 0.0
        lg, wm = runs_of(pops, rng, n_train=1, n_recall=0)[0][4:]
        for k, n in enumerate(RUNS):
            now = 0.0 if k in (4, 8) else 1.0
            if k in (2, 5, 8):
                for q, p in enumerate(projs):
                    si = (rng.random(nets[0].info(f"si_{q}")[1]) < 0.3).astype(np.int8)
                    for net in nets:
                        net.write(f"si_{q}", si)
            logs = []
            for net in nets:
                net.set_stimulus(lg, np.full_like(wm, now))
                net.run(t, n, now, prn)
                logs.append([net.spike_log(p) for p in range(len(pops))] + [net.ss_flags()])
            for p, (a, b) in enumerate(zip(*logs)):
                assert np.array_equal(a, b), f"run {k}: log {p}"
            names = [f"{x}_{p}" for p in range(len(pops)) for x in STATE_POP]
            names += [f"{x}_{q}" for q in range(len(projs))
                      for x in ("pi", "ei", "zi", "ti", "pj", "ej", "zj", "pij", "eij", "zi2", "zj2", "tij", "wij", "qi", "si",
                                ".siq")]
            for name in names:
                a, b = (net.read(name) for net in nets)
                assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), f"run {k}: {name}"
            t, prn = t + n, now
        assert nets[0].counters() == nets[1].counters()
        assert sum(nets[0].counters()) > 0
        if M <= 128:
            assert nets[0].kernel_launches() < nets[1].kernel_launches()
    finally:
        for net in nets:
            net.close()
