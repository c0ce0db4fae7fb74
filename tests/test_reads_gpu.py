"""State reads of 6 to 32 MB: through the driver's copy at first, through
page-locked chunks once they have come to 192 MB, or once a larger read has
allocated the chunks.  The same bytes either way."""
import numpy as np
import pytest

from tests.test_edge_parity_gpu import DT
from tests.test_flow_gpu import pop, proj
from tests.test_gpu_parity import gpu_net

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,reads", [(257, 36), (1023, 11), (1365, 9), (1366, 2)])
def test_repeated_reads(C, reads):
    """48 x 128 x C floats: 6.3, 25, 33.5 and 33.6 MB (32 MiB at C = 1365.3)"""
    rng = np.random.default_rng(C)
    net = gpu_net([pop(48, 128)], [proj(0, 0, C)], DT, seed=1, max_ticks=8)
    try:
        a = rng.integers(0, 2**32, net.info("wij_0")[1], dtype=np.uint32)
        net.write("wij_0", a.view(np.float32))
        for _ in range(reads):
            assert np.array_equal(net.read("wij_0").view(np.uint32), a)
    finally:
        net.close()
