"""The waits of the one-launch closure that run out: with a limit of zero a wait takes one look, so that every
launch of more than one CTA gives up somewhere. The call reports a device error, in every shape of
the kernel, and the GPU, the stream and the workspace serve the next call."""
import pytest
import torch

from scalingelections_b200 import LANES_AUTO, LANES_U16, LANES_U32, _lib, api

pytestmark = pytest.mark.gpu

DEFAULT_NS = 2000000000


@pytest.mark.parametrize("C,lanes", [(129, LANES_U16), (517, LANES_U16), (1024, LANES_U16), (1300, LANES_U16),
                                     (1536, LANES_U16), (700, LANES_U32), (1000, LANES_U32), (1300, LANES_U32),
                                     (600, LANES_AUTO)])
def test_waits_that_run_out(C, lanes):
    g = torch.Generator(device="cuda")
    g.manual_seed(C)
    d = torch.randint(0, 9000, (C, C), generator=g, device="cuda", dtype=torch.int32).view(torch.uint32)
    w = torch.empty(api.closure_workspace_bytes(C, lanes, dataflow=True), dtype=torch.uint8, device="cuda")
    want = api.strongest_paths_device(d, lanes=lanes, workspace=w).view(torch.int32)
    L = _lib.lib()
    L.se_closure_set_wait_limit(0)
    try:
        with pytest.raises(api.SchulzeError) as e:
            api.strongest_paths_device(d, lanes=lanes, workspace=w)
        assert e.value.status == _lib.SE_ERR_DEVICE
        if lanes != LANES_AUTO:
            api.strongest_paths_enqueue(d, lanes=lanes, workspace=w)
            with pytest.raises(api.SchulzeError) as e:
                api.closure_check(w)
            assert e.value.status == _lib.SE_ERR_DEVICE
    finally:
        L.se_closure_set_wait_limit(DEFAULT_NS)
    for _ in range(3):
        assert torch.equal(api.strongest_paths_device(d, lanes=lanes, workspace=w).view(torch.int32), want)
    assert api.last_closure_schedule() == api.CLOSURE_RESIDENT
