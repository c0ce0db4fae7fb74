"""Calls whose route depends on a size, at the sizes where it changes: reads
through page-locked memory (6 and 24 MB), a run's begin (8 populations and
projections in one launch), a stimulus row (448 HCUs passed by value), the
column parts of the BF16 recall contraction (tiles against 148 SMs), the
exponentials of the recall's population update away from its usual range, and
the delay queue as bit planes for every queue word."""
import numpy as np
import pytest

from tests.test_edge_parity_gpu import DT
from tests.test_flow_gpu import pop, proj
from tests.test_gpu_parity import gpu_net
from tests.test_recall_gpu import Pop, bits_equal

pytestmark = pytest.mark.gpu

f32 = np.float32


@pytest.mark.parametrize("C", [1, 255, 256, 257, 1023, 1024, 1025, 1500])
def test_reads(C):
    """48 x 128 x C floats: 6 MB at C = 256, 24 MB at 1024"""
    rng = np.random.default_rng(C)
    net = gpu_net([pop(48, 128)], [proj(0, 0, C)], DT, seed=1, max_ticks=8)
    try:
        for name in ("wij_0", "pij_0"):
            a = rng.integers(0, 2**32, net.info(name)[1], dtype=np.uint32)
            net.write(name, a.view(f32))
            # the allocation-free read takes cell fields of at most 2^20 elements
            for read in (net.read, net.read_noalloc) if name == "wij_0" or a.size <= 1 << 20 else (net.read,):
                assert np.array_equal(read(name).view(np.uint32), a)
    finally:
        net.close()


@pytest.mark.parametrize("n", [7, 8, 9])
def test_run_begin(n):
    """n populations of their own projection each: the first 7 do not depend on n"""
    rng = np.random.default_rng(5)
    conn = [rng.choice(60, 40).astype(np.int32) for _ in range(9)]
    nets = []
    try:
        for k in (7, n):
            net = gpu_net([pop(2, 30)] * k, [proj(q, q, 20) for q in range(k)], DT, seed=3, poisson_hz=40.0, max_ticks=32)
            nets.append(net)
            for q in range(k):
                net.set_conn(q, conn[q], np.full(40, 1 + q, np.int32))
            net.set_stimulus(np.zeros(60 * k, f32), np.ones(2 * k, f32))
            for first, ticks, prn, old in ((1, 20, 1.0, 0.0), (21, 32, 0.0, 1.0), (53, 9, 1.0, 0.0)):
                net.run(first, ticks, prn, old)
        for q in range(7):
            assert np.array_equal(nets[0].spike_log(q), nets[1].spike_log(q))
            for x in ("dsup", "epsc", "bj", "pi", "pij", "wij", "tij", "qi"):
                a, b = (net.read(f"{x}_{q}") for net in nets)
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (x, q)
    finally:
        for net in nets:
            net.close()


@pytest.mark.parametrize("H", [1, 448, 449])
def test_stimulus_row(H):
    """the row of set_stimulus_idx against the same row of an uploaded table"""
    rng = np.random.default_rng(H)
    lg = rng.integers(-1, 5, H).astype(np.int32)
    wm = rng.random(H).astype(f32)
    nets = [gpu_net([pop(H, 5)], [proj(0, 0, 5)], DT, seed=2, max_ticks=8) for _ in range(2)]
    try:
        nets[0].set_stimulus_idx(lg, 1e-4, wm)
        nets[1].upload_stimuli_idx(lg[None], 1e-4, wm[None])
        nets[1].use_stimulus(0, 0)
        for net in nets:
            net.run(1, 3, 1.0, 1.0)
        assert bits_equal(nets[0].read("dsup_0"), nets[1].read("dsup_0"))
        assert np.array_equal(nets[0].spike_log(0), nets[1].spike_log(0))
    finally:
        for net in nets:
            net.close()


def test_recall_column_parts():
    """a replicate does not depend on how many there are: 8, 4, 2 parts and none per tile, against 149 tiles"""
    H, M, big = 8, 32, 149
    rng = np.random.default_rng(11)
    p = Pop(H, M, hz=60.0)
    N, R = p.N, 128 * big
    W, vec = rng.standard_normal((N, N)) * 0.5, rng.standard_normal((3, N))
    lg, wm = rng.integers(-1, M, (R, H)), (rng.random((R, H)) < 0.5).astype(f32)
    hist = [(rng.random((R, N)) < 0.1).astype(np.int8) for _ in range(3)]
    want = None
    for tiles in (big, 1, 18, 19, 37, 38, 74, 75):
        r = 128 * tiles
        eng = p.engine(r)
        eng.load_state(W, *vec, *np.zeros((3, N)))
        eng.set_cues(lg[:r], p.eps, wm[:r])
        for name, s in zip(("spike_tm3", "spike_tm2", "spike_tm1"), hist):
            eng.write(name, s[:r])
        eng.run(10, 5)
        got = [eng.read(x) for x in ("epsc", "dsup", "spike")]
        eng.close()
        want = want or got
        for a, b in zip(got, want):
            assert np.array_equal(a.view(np.uint8), b[:r].view(np.uint8)), tiles


@pytest.mark.parametrize("M", [16, 64])
@pytest.mark.parametrize("more", [dict(wtagain=60.0), dict(lgbias=-40.0), dict(lgbias=-1.0, wtagain=0.01),
                                  dict(lgbias=120.0, wtagain=3.0)])
def test_recall_population_range(M, more):
    """exponentials that underflow, sums of at most 1, and a maximum that overflows, bit for bit"""
    H, R = 512 // M, 128
    rng = np.random.default_rng(M)
    p = Pop(H, M, **more)
    N = p.N
    bj = (rng.standard_normal(N) * 3).astype(f32)
    lg, wm = rng.integers(-1, M, (R, H)).astype(np.int32), (rng.random((R, H)) < 0.7).astype(f32)
    eng = p.engine(R)
    eng.load_state(rng.standard_normal((N, N)), bj, rng.standard_normal(N) * 3, rng.standard_normal(N) * 9, *np.zeros((3, N)))
    eng.set_cues(lg, p.eps, wm)
    for t in range(10, 14):
        dsup, epsc = eng.read("dsup"), eng.read("epsc")
        eng.run(t, 1)
        with np.errstate(all="ignore"):
            want, spk = p.update(dsup, epsc, bj, lg, wm, t)
        assert bits_equal(eng.read("dsup"), want)
        assert np.array_equal(eng.read("spike"), spk)
    eng.close()


@pytest.mark.parametrize("M,C", [(10, 63), (10, 64), (10, 65), (40, 129), (10, 2100)])
def test_queue_words(M, C):
    """every delay, and queue words of any bits, the sign included, which its shift repeats"""
    H = 5 if C < 1000 else 21
    rng = np.random.default_rng(M * 1000 + C)
    nets = [gpu_net([pop(H, M)], [proj(0, 0, min(C, H * M))], DT, seed=9, poisson_hz=30.0, max_ticks=80, per_tick=t)
            for t in (False, True)]
    try:
        n = nets[0].info("qi_0")[1]
        ii = rng.integers(-1, H * M, n).astype(np.int32)
        di = rng.integers(1, 32, n).astype(np.int32)
        qi = (rng.integers(0, 2**32, n, dtype=np.uint32) & rng.integers(0, 2**32, n, dtype=np.uint32)).view(np.int32)
        qi[rng.random(n) < 0.7] = 0
        for net in nets:
            net.set_conn(0, ii, di)
            net.set_stimulus(np.zeros(H * M, f32), np.ones(H, f32))
            net.write("qi_0", qi)
        t = 1
        for ticks in (1, 2, 31, 32, 33, 7, 80):
            for net in nets:
                net.run(t, ticks, 1.0, 1.0)
            t += ticks
            for x in ("qi_0", ".siq_0", "epsc_0", "pi_0", "wij_0"):
                a, b = (net.read(x) for net in nets)
                assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), (x, t)
            assert np.array_equal(nets[0].spike_log(0), nets[1].spike_log(0))
    finally:
        for net in nets:
            net.close()
