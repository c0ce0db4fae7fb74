"""The FP32 contraction of the replicate recall engine, by events and dense:
epsc bit-identical to the float32 sum of the spiking sources' weights in
ascending source order, which is what the engine's FP32 form defines.

The shapes cross the event kernel's edges: chunks of 384 sources (256: one
partial chunk; 512: a second chunk of one box; 1024: three), passes of 360
replicates, spike counts per chunk around and above the listed 32, rows of no
spikes and of all, and the two reasons for the dense kernel (many spikes by
the population's rates, a weight that is not finite)."""
import numpy as np
import pytest

from tests.test_recall_gpu import Pop, bits_equal

pytestmark = pytest.mark.gpu

f32 = np.float32


def ordered_sum(epsc, s, W, kepsc):
    acc = np.zeros_like(epsc)
    with np.errstate(invalid="ignore"):
        for i in range(W.shape[0]):
            rows = s[:, i] != 0
            acc[rows] += W[i]
    return epsc * (f32(1) - f32(kepsc)) + acc


def engine(H, M, R, hz, rng, W):
    pop = Pop(H, M, hz=hz)
    N = pop.N
    eng = pop.engine(R, "fp32")
    eng.load_state(W, rng.standard_normal(N), rng.standard_normal(N), rng.standard_normal(N) - 3, *np.zeros((3, N)))
    lgidx = rng.integers(-1, M, (R, H)).astype(np.int32)
    eng.set_cues(lgidx, pop.eps, (rng.random((R, H)) < 0.5).astype(f32))
    return pop, eng


@pytest.mark.parametrize("H,M,R,hz", [(16, 16, 128, 20.0), (8, 64, 640, 0.0), (32, 32, 384, 40.0), (16, 64, 128, 180.0),
                                      (16, 16, 128, 300.0)])
def test_epsc_bits(H, M, R, hz):
    rng = np.random.default_rng(H * 100 + M + int(hz))
    N = H * M
    W = (rng.standard_normal((N, N)) * 0.5).astype(f32)
    pop, eng = engine(H, M, R, hz, rng, W)
    # per-replicate histories: 2% spikes, around the list capacity of a chunk, and rows of none, of all, of one
    hist = []
    for dens in (0.02, 32 / 384, 0.5):
        s = (rng.random((R, N)) < dens).astype(np.int8)
        s[0], s[1], s[2] = 0, 1, 0
        s[2, N - 1] = 1
        hist.append(s)
    for name, s in zip(("spike_tm3", "spike_tm2", "spike_tm1"), hist):
        eng.write(name, s)
        assert np.array_equal(eng.read(name), s)
    epsc = eng.read("epsc")
    for t in range(10, 15):
        eng.run(t, 1)
        epsc = ordered_sum(epsc, hist[-3], W, pop.kepsc)
        assert bits_equal(eng.read("epsc"), epsc), f"tick {t}"
        hist.append(eng.read("spike"))
    eng.close()


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_weight_not_finite(value):
    """0 * w is NaN for such a weight: its whole column is, whatever spikes"""
    H, M, R = 8, 32, 128
    rng = np.random.default_rng(3)
    W = (rng.standard_normal((H * M, H * M)) * 0.5).astype(f32)
    W[17, 5] = value
    pop, eng = engine(H, M, R, 20.0, rng, W)
    epsc = eng.read("epsc")
    eng.run(10, 1)
    got = eng.read("epsc")
    assert np.all(np.isnan(got[:, 5]))
    keep = np.arange(H * M) != 5
    assert bits_equal(got[:, keep], ordered_sum(epsc, np.zeros((R, H * M)), W, pop.kepsc)[:, keep])
    eng.close()
