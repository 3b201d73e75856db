"""The one-launch closure where its CTAs are not all on the GPU in time: it gives way before it writes
anything, and the launches close the matrix instead, for calls that wait and calls that only queue.
A limit of zero makes every launch of more than one CTA give way."""
import numpy as np
import pytest
import torch

from scalingelections_b200 import LANES_AUTO, LANES_U16, LANES_U32, _lib, api
from scalingelections_b200.batch import BatchedElections

pytestmark = pytest.mark.gpu

DEFAULT_NS = 1000000
KINDS = [(LANES_U16, 0, 9000), (LANES_U32, 0, 2**32), (LANES_AUTO, 0, 9000), (LANES_AUTO, 0, 2**32),
         (LANES_AUTO, 70000, 130000)]


@pytest.fixture
def always_gives_way():
    _lib.lib().se_closure_set_start_limit(0)
    yield
    _lib.lib().se_closure_set_start_limit(DEFAULT_NS)


def matrix(C, lo, hi, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randint(lo, hi, (C, C), generator=g, device="cuda", dtype=torch.int64).to(torch.int32).view(torch.uint32)


def by_rounds(d, lanes):
    api.set_closure_mode(1)
    try:
        return api.strongest_paths_device(d, lanes=lanes).view(torch.int32)
    finally:
        api.set_closure_mode(0)


def enqueue(d, lanes, out=None):
    w = torch.empty(api.closure_workspace_bytes(d.shape[0], lanes, dataflow=True), dtype=torch.uint8, device="cuda")
    out = api.strongest_paths_enqueue(d, lanes=lanes, out=out, workspace=w)
    return w, out


@pytest.mark.parametrize("C", [64, 65, 128, 129, 300, 517, 769, 1025, 1089, 1344, 1536])
def test_results_after_giving_way(always_gives_way, C):
    for lanes, lo, hi in KINDS:
        d = matrix(C, lo, hi, seed=C + lanes)
        want = by_rounds(d, lanes)
        assert torch.equal(api.strongest_paths_device(d, lanes=lanes).view(torch.int32), want), (lanes, hi)
        assert (api.last_closure_schedule() == api.CLOSURE_RESIDENT) == (C == 64)
        if lanes != LANES_AUTO:
            w, out = enqueue(d, lanes)
            api.closure_check(w)
            assert torch.equal(out.view(torch.int32), want), (lanes, hi)
        api.strongest_paths_device(d, lanes=lanes, out=d)  # over its input
        assert torch.equal(d.view(torch.int32), want), (lanes, hi)


@pytest.mark.parametrize("lanes", [LANES_U16, LANES_U32])
def test_queued_over_the_input_and_with_odd_strides(always_gives_way, lanes):
    C = 700
    big = torch.full((C, C + 3), -1, dtype=torch.int32, device="cuda")
    big[:, :C] = matrix(C, 0, 9000, seed=5).view(torch.int32)
    d = big.view(torch.uint32)[:, :C]
    want = by_rounds(d, lanes)
    w, _ = enqueue(d, lanes, out=d)
    api.closure_check(w)
    assert torch.equal(big[:, :C], want) and bool((big[:, C:] == -1).all())


def test_overflow_after_giving_way(always_gives_way):
    d = matrix(300, 0, 200000, seed=1)
    with pytest.raises(api.SchulzeError, match="65535"):
        api.strongest_paths_device(d, lanes=LANES_U16)
    w, _ = enqueue(d, LANES_U16)
    with pytest.raises(api.SchulzeError, match="65535"):
        api.closure_check(w)


def test_the_limit_belongs_to_the_thread(always_gives_way):
    import threading

    ran = []

    def other():
        api.strongest_paths_device(matrix(300, 0, 9000, seed=2), lanes=LANES_U16)
        ran.append(api.last_closure_schedule())

    t = threading.Thread(target=other)
    t.start()
    t.join()
    assert ran == [api.CLOSURE_RESIDENT]


def test_beside_a_persistent_batch():
    """A batch on another stream holds every SM for some tens of milliseconds: closures queued and
    waited for meanwhile are right in whatever form they run."""
    sizes = [1000, 600, 500, 400] * 60
    batch = BatchedElections([matrix(C, 0, 5000, seed=i) for i, C in enumerate(sizes)], [LANES_U16] * len(sizes),
                             ctas_per_sm=2)
    batch.run()
    batch.check()
    first = [s.clone() for s in batch.strongest_paths]
    mats = [(C, lanes, matrix(C, 0, 9000, seed=C)) for C in (300, 1024, 1300) for lanes in (LANES_U16, LANES_U32)]
    want = [by_rounds(d, lanes) for _, lanes, d in mats]
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    batch.run()
    with torch.cuda.stream(other):
        queued = [enqueue(d, lanes) for _, lanes, d in mats]
        waited = [api.strongest_paths_device(d, lanes=lanes) for _, lanes, d in mats]
        for w, _ in queued:
            api.closure_check(w)
    batch.check()
    for (C, lanes, _), ref, (_, q), s in zip(mats, want, queued, waited):
        assert torch.equal(q.view(torch.int32), ref) and torch.equal(s.view(torch.int32), ref), (C, lanes)
    for a, b in zip(batch.strongest_paths, first):
        assert np.array_equal(a.view(torch.int32).cpu().numpy(), b.view(torch.int32).cpu().numpy())
