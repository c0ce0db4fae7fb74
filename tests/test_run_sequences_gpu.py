"""Runs that do not follow each other as a plain schedule's do, bit for bit
against the path of one launch per tick: external spikes set between runs, which
take a network from the dataflow kernel to the kernels with a grid barrier with
the list, the queue and the spike buffers that the other one left; a run whose
first tick is later or earlier than the one after the last; decay tables built
in FP64; and networks whose HCUs are too large for the dataflow kernel, over
several column units."""
import numpy as np
import pytest

from tests.harness import STATE_POP
from tests.test_edge_parity_gpu import DT
from tests.test_flow_gpu import network, pop, proj
from tests.test_flow_state_gpu import same
from tests.test_gpu_parity import gpu_net

pytestmark = pytest.mark.gpu


class Pair:
    """two networks of the same tables and stimulus, by the default path and by one launch per tick"""

    def __init__(self, pops, projs, seed, variant=0, connected=0.9, **kw):
        rng = self.rng = np.random.default_rng(seed)
        if variant:
            pops = [dict(p, taua=0.05, adgain=1.0) for p in pops]
            kw.update(variant=1, spike_buffer=kw.get("spike_buffer", 25))
        self.nets = [gpu_net(pops, projs, DT, seed=4, poisson_hz=40.0, max_ticks=64, per_tick=p, **kw) for p in (False, True)]
        self.pops, self.projs, self.variant, self.prn = pops, projs, variant, 0.0
        for q, p in enumerate(projs):
            n, ns = self.nets[0].info(f"ii_{q}")[1], pops[p["src_pop"]]["hcu_num"] * pops[p["src_pop"]]["mcu_num"]
            ii = np.where(rng.random(n) < connected, rng.integers(0, ns, n), -1).astype(np.int32)
            di = rng.integers(1, 6, n).astype(np.int32)
            for net in self.nets:
                net.set_conn(q, ii, di)
        self.n = [p["hcu_num"] * p["mcu_num"] for p in pops]
        lg = (rng.random(sum(self.n)) * 3 - 3).astype(np.float32)
        for net in self.nets:
            net.set_stimulus(lg, np.ones(sum(p["hcu_num"] for p in pops), np.float32))

    def run(self, first, n, prn, what):
        logs = []
        for net in self.nets:
            net.run(first, n, prn, self.prn)
            logs.append([net.spike_log(p) for p in range(len(self.pops))] + [net.ss_flags()])
        self.prn = prn
        for a, b in zip(*logs):
            assert np.array_equal(a, b), f"{what}: logs"
        names = [f"{x}_{p}" for p in range(len(self.pops)) for x in (*STATE_POP, *(("ada",) if self.variant else ()))]
        names += [f"{x}_{q}" for q in range(len(self.projs))
                  for x in ("pi", "ei", "zi", "ti", "pj", "ej", "zj", "pij", "eij", "zj2", "wij", "qi", "si", ".siq",
                            *(() if self.variant else ("zi2", "tij")))]
        same(self.nets, names, what)

    def close(self):
        assert self.nets[0].counters() == self.nets[1].counters() and sum(self.nets[0].counters()) > 0
        for net in self.nets:
            net.close()


@pytest.mark.parametrize("variant,H,M,C,H0", [(0, 7, 30, 77, 0), (0, 5, 65, 130, 3), (0, 152, 20, 41, 0), (1, 7, 30, 77, 0),
                                              (1, 5, 65, 130, 0)])
def test_external_spikes_between_runs(variant, H, M, C, H0):
    pair = Pair(*network(H, M, C, H0), seed=H, variant=variant)
    assert pair.nets[0].run_form()[0] == "dataflow"
    t = 1
    for n in (3, 1, 6, 2):
        pair.run(t, n, 1.0, f"before, from {t}")
        t += n
    for p in range(len(pair.pops)):
        table = {k: pair.rng.choice(pair.n[p], 2, replace=False).tolist() for k in range(t, t + 40)}
        for net in pair.nets:
            net.set_ext_spikes(p, table)
        assert pair.nets[0].run_form()[0] == "barrier"
        for n, prn in ((1, 1.0), (5, 1.0), (2, 0.0), (4, 1.0)):
            pair.run(t, n, prn, f"population {p} replayed, from {t}")
            t += n
    pair.close()


@pytest.mark.parametrize("variant,H,M,C,H0,ring", [(0, 6, 31, 80, 0, 1), (0, 4, 70, 150, 3, 1), (1, 6, 31, 80, 0, 25),
                                                   (1, 4, 70, 150, 0, 32), (1, 6, 31, 80, 0, 3)])
def test_ticks_skipped_and_repeated(variant, H, M, C, H0, ring):
    """cells and rows with a later tick than the run's first take no decay (ProcUpdMulti: gsbn's expressions for a
    negative number of ticks); a gap decays them over it, and may be longer than the ring"""
    pair = Pair(*network(H, M, C, H0), seed=H + ring, variant=variant, spike_buffer=ring)
    assert pair.nets[0].run_form()[0] == "dataflow"
    for first, n, prn in ((1, 6, 1.0), (9, 5, 1.0), (60, 4, 1.0), (61, 5, 1.0), (63, 2, 1.0), (30, 8, 1.0), (38, 1, 0.0),
                          (39, 3, 0.0), (20, 3, 0.0), (2000, 5, 1.0), (2005, 6, 1.0)):
        pair.run(first, n, prn, f"from {first}")
    pair.close()


@pytest.mark.parametrize("H,M,C,H0", [(5, 20, 60, 0), (4, 100, 300, 3), (150, 33, 40, 0)])
def test_fp64_tables(H, M, C, H0):
    pair = Pair(*network(H, M, C, H0), seed=H + M, fp64_tables=1)
    assert pair.nets[0].run_form()[0] == "dataflow"
    t = 1
    for n, prn in ((4, 1.0), (1, 1.0), (33, 1.0), (7, 0.0), (20, 1.0)):
        pair.run(t, n, prn, f"from {t}")
        t += n
    pair.close()


@pytest.mark.parametrize("H,M,C,threads", [(6, 129, 700, 512), (6, 129, 700, 256), (4, 256, 1024, 512), (4, 256, 1024, 256),
                                           (148, 130, 260, 512), (160, 140, 300, 256), (3, 512, 1536, 512)])
def test_hcus_beyond_the_dataflow_kernel(H, M, C, threads):
    pair = Pair([pop(H, M)], [proj(0, 0, C)], seed=M, tick_threads=256 if threads == 256 and H < 149 else 0)
    assert pair.nets[0].run_form() == ("barrier", threads)
    t = 1
    for n, prn in ((1, 1.0), (2, 1.0), (30, 1.0), (5, 0.0), (3, 1.0)):
        pair.run(t, n, prn, f"from {t}")
        t += n
    pair.close()
