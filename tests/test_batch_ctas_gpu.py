"""CTAs per SM of a batch that leaves them open: each of its persistent launches by its own tasks and chain."""
import pytest
import torch

from scalingelections_b200 import LANES_U16, LANES_U32
from scalingelections_b200.batch import BatchedElections

pytestmark = pytest.mark.gpu

CHAIN, MANY = [1700] * 3, [140 + 5 * (n % 30) for n in range(600)]  # few tasks for a long chain; the opposite


def ctas(parts, ctas_per_sm=0):
    """parts: (sizes, lanes, micro-tile)."""
    prefs = {C: torch.zeros((C, C), dtype=torch.int32, device="cuda").view(torch.uint32) for p in parts for C in p[0]}
    flat = [(prefs[C], lanes, micro) for sizes, lanes, micro in parts for C in sizes]
    b = BatchedElections([f[0] for f in flat], [f[1] for f in flat], ranking=False, ctas_per_sm=ctas_per_sm,
                         micro_tiles=[f[2] for f in flat])
    try:
        return b.cta_counts()
    finally:
        b.close()


def test_each_launch_by_its_own():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert ctas([(CHAIN, LANES_U16, 8)]) == (sms, 0, 0)
    assert ctas([(MANY, LANES_U16, 8)]) == (2 * sms, 0, 0)
    assert ctas([(CHAIN, LANES_U16, 8), (MANY, LANES_U16, 4)]) == (sms, 0, 2 * sms)
    assert ctas([(MANY, LANES_U16, 8), (CHAIN, LANES_U16, 4)]) == (2 * sms, 0, sms)
    assert ctas([(CHAIN, LANES_U16, 8), (MANY, LANES_U32, 8)]) == (sms, sms, 0)
    assert ctas([(CHAIN, LANES_U16, 8), (MANY, LANES_U16, 4)], 99) == (2 * sms, 0, 2 * sms)
    assert ctas([([100] * 1000, LANES_U16, 8)]) == (2 * sms, 0, 0)
    assert ctas([(CHAIN, LANES_U16, 8), (MANY, LANES_U16, 4)], 1) == (sms, 0, sms)
    assert ctas([([20], LANES_U16, 8)]) == (1, 0, 0)
