"""The one-launch closure of small matrices (the automatic schedule with a full workspace) against
the round-by-round schedule and, where it is quick, the oracle: sizes on both sides of each block,
round and tile-shape limit, every lane mode, a shifted 16-bit window, values that need 32 bits in the
automatic mode, odd strides, an output over its own input, and closures on two streams at once."""
import numpy as np
import pytest
import torch

from scalingelections_b200 import LANES_AUTO, LANES_U16, LANES_U32, api

pytestmark = pytest.mark.gpu


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


@pytest.mark.parametrize("C", [1, 3, 32, 33, 64, 65, 96, 97, 129, 257, 768, 769, 1024, 1025, 1088, 1089, 1344, 1345,
                               1536, 1537])
def test_sizes_and_lanes(orc, C):
    for lanes, lo, hi in ((LANES_U16, 0, 9000), (LANES_U32, 0, 2**32), (LANES_AUTO, 0, 9000), (LANES_AUTO, 0, 2**32),
                          (LANES_AUTO, 70000, 130000)):
        d = matrix(C, lo, hi, seed=C + lanes)
        got = api.strongest_paths_device(d, lanes=lanes).view(torch.int32)
        assert torch.equal(got, by_rounds(d, lanes)), (lanes, hi)
        if C <= 257:
            P = api._to_host_u32(d)
            assert np.array_equal(api._to_host_u32(got.view(torch.uint32)), orc.strongest_paths(P, "blocked", tile=16))


def test_sixteen_bit_overflow_is_reported():
    with pytest.raises(api.SchulzeError, match="65535"):
        api.strongest_paths_device(matrix(300, 0, 200000, seed=1), lanes=LANES_U16)


@pytest.mark.parametrize("C,ld,ldo", [(130, 131, 133), (517, 520, 517), (1100, 1102, 1101)])
def test_strides(C, ld, ldo):
    big = torch.zeros((C, ld), dtype=torch.int32, device="cuda")
    big[:, :C] = matrix(C, 0, 9000, seed=C).view(torch.int32)
    d = big.view(torch.uint32)[:, :C]
    out = torch.full((C, ldo), -1, dtype=torch.int32, device="cuda")
    api.strongest_paths_device(d, lanes=LANES_U16, out=out.view(torch.uint32)[:, :C])
    assert torch.equal(out[:, :C], by_rounds(d.contiguous(), LANES_U16))
    assert bool((out[:, C:] == -1).all())


@pytest.mark.parametrize("C", [100, 700, 1500])
def test_output_over_the_input(C):
    d = matrix(C, 0, 9000, seed=C)
    want = by_rounds(d, LANES_U16)
    api.strongest_paths_device(d, lanes=LANES_AUTO, out=d)
    assert torch.equal(d.view(torch.int32), want)


def test_two_streams():
    """Queued alternately on two streams without a wait between them: launches that fill the GPU
    and ones that do not."""
    sizes = [768, 1088, 300, 1500, 64, 1024]
    mats = [matrix(C, 0, 9000, seed=C) for C in sizes]
    want = [by_rounds(d, LANES_U16) for d in mats]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    jobs = []
    for n in range(4 * len(sizes)):
        d = mats[n % len(sizes)]
        with torch.cuda.stream(streams[n % 2]):
            w = torch.empty(api.closure_workspace_bytes(d.shape[0], LANES_U16, dataflow=True), dtype=torch.uint8,
                            device="cuda")
            jobs.append((w, streams[n % 2], api.strongest_paths_enqueue(d, lanes=LANES_U16, workspace=w)))
    for n, (w, s, out) in enumerate(jobs):
        with torch.cuda.stream(s):
            api.closure_check(w)
        assert torch.equal(out.view(torch.int32), want[n % len(sizes)])
