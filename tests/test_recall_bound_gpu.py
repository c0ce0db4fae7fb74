"""The recall's population update divides an activity by the HCU's sum only
where a uniform is near the product that decides a spike.  Where the sum is near
the largest float (a negative wtagain, and a support 88.7 below the others'),
uniforms just below that product: each is a spike.  Bit for bit against the
float32 restatement, as the tests of the usual range."""
import numpy as np
import pytest

from tests.test_recall_gpu import Pop, bits_equal

pytestmark = pytest.mark.gpu

# ticks at which one of 128 x 4 HCUs' uniforms lies within 2e-4 of the product, relative to it, from below
TICKS = (15743, 18114, 38647, 49700, 51957, 65856)


@pytest.mark.parametrize("contraction", ["bf16", "fp32"])
def test_sums_near_the_largest_float(contraction):
    H, M, R, J = 4, 64, 128, 5
    p = Pop(H, M, wtagain=-1.0, maxfq=1.0, taum=1e6, hz=0.0, lgbias=0.0)
    N = p.N
    dsup, zero = np.zeros((H, M), np.float32), np.zeros(N, np.float32)
    dsup[:, J] = -88.66479
    lg, wm = np.full((R, H), -1, np.int32), np.zeros((R, H), np.float32)
    eng = p.engine(R, contraction)
    for tick in TICKS:
        eng.load_state(np.zeros((N, N), np.float32), zero, zero, dsup.reshape(-1), *np.zeros((3, N)))
        eng.set_cues(lg, p.eps, wm)
        eng.run(tick, 1)
        with np.errstate(all="ignore"):
            want, spk = p.update(np.tile(dsup.reshape(1, -1), (R, 1)), np.zeros((R, N), np.float32), zero, lg, wm, tick)
        assert bits_equal(eng.read("dsup"), want)
        assert np.array_equal(eng.read("spike"), spk)
        assert spk[:, J::M].any()
    eng.close()
