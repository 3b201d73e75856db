"""Which form of the closure a call takes: the one-launch closure in registers or the launches, as the
host query predicts it and as the last call of the thread reports it."""
import numpy as np
import pytest
import torch

from scalingelections_b200 import LANES_AUTO, LANES_U16, LANES_U32, _lib, api

# (lanes, largest size that fits the register files)
LIMITS = [(LANES_U16, 1536), (LANES_U32, 1344)]


@pytest.mark.parametrize("lanes,limit", LIMITS)
def test_query_at_the_size_limit(lanes, limit):
    assert api.closure_is_resident(1, lanes) and api.closure_is_resident(limit, lanes)
    assert not api.closure_is_resident(limit + 1, lanes)
    assert not api.closure_is_resident(0, lanes)
    assert not api.closure_is_resident(1000, lanes, api.closure_workspace_bytes(1000, lanes))  # the plain workspace
    api.set_closure_mode(1)
    try:
        assert not api.closure_is_resident(1000, lanes)
    finally:
        api.set_closure_mode(0)


def test_launch_count_counts_the_form_that_runs():
    L = _lib.lib()
    assert L.se_closure_launch_count(1536) == 1
    assert L.se_closure_launch_count(1537) == 3 + 13 + 1  # 13 pivot rounds, one launch per round
    api.set_closure_mode(1)
    try:
        assert L.se_closure_launch_count(1536) == 3 + 2 * 12
    finally:
        api.set_closure_mode(0)


def closure(C, lanes, lo=0, hi=9000, **kw):
    d = api._to_device_u32(np.random.default_rng(C).integers(lo, hi, size=(C, C), dtype=np.uint64).astype(np.uint32), "cuda")
    api.strongest_paths_device(d, lanes=lanes, **kw)
    return api.last_closure_schedule()


@pytest.mark.gpu
@pytest.mark.parametrize("lanes,limit", LIMITS)
def test_form_that_ran(lanes, limit):
    assert closure(limit, lanes) == api.CLOSURE_RESIDENT
    assert closure(limit + 1, lanes) == api.closure_schedule(limit + 1, lanes)
    plain = torch.empty(api.closure_workspace_bytes(limit, lanes), dtype=torch.uint8, device="cuda")
    assert closure(limit, lanes, workspace=plain) == 1
    api.set_closure_mode(3)
    try:
        assert closure(limit, lanes) == (3 if lanes == LANES_U16 else 1)
    finally:
        api.set_closure_mode(0)


@pytest.mark.gpu
def test_form_that_ran_with_automatic_lanes():
    assert closure(1536, LANES_AUTO) == api.CLOSURE_RESIDENT
    assert closure(1344, LANES_AUTO, hi=2**32) == api.CLOSURE_RESIDENT  # again in 32-bit lanes
    assert closure(1345, LANES_AUTO, hi=2**32) == api.closure_schedule(1345, LANES_U32)
