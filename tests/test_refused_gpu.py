"""A call that CUDA refuses is reported once: the runtime's own record of it
does not fail the next network."""
import pytest

from gsbn_b200 import capi
from tests.test_edge_parity_gpu import DT
from tests.test_flow_gpu import pop, proj

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1])
def test_networks_too_large_for_shared_memory(variant):
    """slots per HCU through the sizes where first CUDA refuses the shared memory and then the library does"""
    more = dict(variant=1, spike_buffer=25) if variant else {}
    pops = [dict(p, taua=0.05, adgain=1.0) if variant else p for p in (pop(300, 70), pop(1, 70))]
    status = set()
    for C in range(8600, 9000, 8):
        try:
            capi.Net(pops, [proj(0, 1, C)], DT, seed=1, max_ticks=8, **more).close()
            status.add(0)
        except capi.BcpnnError as e:
            status.add(e.status)
            net = capi.Net([pops[1]], [proj(0, 0, 70)], DT, seed=1, max_ticks=8, **more)
            net.run(1, 3, 1.0, 1.0)
            net.sync()
            net.close()
    assert -2 in status and len(status) > 1, status
