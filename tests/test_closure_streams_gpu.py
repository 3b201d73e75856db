"""The one-launch closure on several streams and threads: two that do not fit the GPU together are never
both made, ones that fit run side by side, and no call waits for another stream's work."""
import threading

import pytest
import torch

from scalingelections_b200 import LANES_U16, LANES_U32, _lib, api

pytestmark = pytest.mark.gpu

PER_THREAD = 2  # cudaStreamPerThread: one handle, another stream in every thread
LONG = 600_000_000  # cycles of a stream's earlier work: about 0.3 s


def matrix(C, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randint(0, 9000, (C, C), generator=g, device="cuda", dtype=torch.int32).view(torch.uint32)


def by_rounds(d, lanes):
    api.set_closure_mode(1)
    try:
        return api.strongest_paths_device(d, lanes=lanes).view(torch.int32)
    finally:
        api.set_closure_mode(0)


class Job:
    """One closure with buffers of its own, so that nothing is allocated while streams run."""

    def __init__(self, C, lanes=LANES_U16):
        self.d, self.lanes, self.C = matrix(C, C), lanes, C
        self.want = by_rounds(self.d, lanes)
        self.out = torch.empty_like(self.d)
        self.work = torch.empty(api.closure_workspace_bytes(C, lanes, dataflow=True), dtype=torch.uint8, device="cuda")

    def enqueue(self):
        api.strongest_paths_enqueue(self.d, lanes=self.lanes, out=self.out, workspace=self.work)
        return api.last_closure_schedule()

    def right(self):
        api.closure_check(self.work)
        return torch.equal(self.out.view(torch.int32), self.want)


def test_two_threads_on_their_per_thread_streams():
    sizes = [(1024, LANES_U16), (1300, LANES_U16), (1000, LANES_U32), (700, LANES_U16), (300, LANES_U16)]
    jobs = [[Job(C, lanes) for C, lanes in sizes] for _ in range(2)]
    torch.cuda.synchronize()
    failed = []

    def work(mine):
        L = _lib.lib()
        torch.cuda.set_device(0)
        for _ in range(20):
            for j in mine:
                st = L.se_closure(j.d.data_ptr(), j.C, j.C, j.out.data_ptr(), j.C, j.lanes, 0, j.work.data_ptr(),
                                  j.work.numel(), PER_THREAD)
                if st:
                    failed.append((j.C, st, _lib.last_error()))

    threads = [threading.Thread(target=work, args=(mine,)) for mine in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed
    assert all(torch.equal(j.out.view(torch.int32), j.want) for mine in jobs for j in mine)


@pytest.mark.parametrize("C", [60, 300, 1024, 1500])
def test_a_call_does_not_wait_for_another_stream(C):
    a, b = Job(C), Job(C)
    A, B = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(A):
        torch.cuda._sleep(LONG)
        a.enqueue()
    with torch.cuda.stream(B):
        b.enqueue()
        B.synchronize()
        assert not A.query()  # A's closure is still behind its earlier work
        assert b.right()
    with torch.cuda.stream(A):
        assert a.right()


def test_closures_in_flight_share_the_gpu_where_they_fit():
    """Queued while another stream's closure is in flight: 25 CTAs beside 25 of another stream are
    resident, 256 are not; after a stream's closures of its own, and once the other is done, they are."""
    a, b, big, again = Job(300), Job(300), Job(1024), Job(1024)
    A, B = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(A):
        torch.cuda._sleep(LONG)
        assert a.enqueue() == api.CLOSURE_RESIDENT
    with torch.cuda.stream(B):
        assert b.enqueue() == api.CLOSURE_RESIDENT
        assert big.enqueue() == api.closure_schedule(1024)
        assert not A.query()
        assert b.right() and big.right()
    with torch.cuda.stream(A):
        assert again.enqueue() == api.CLOSURE_RESIDENT  # its own stream's come one after another
        assert a.right() and again.right()
    with torch.cuda.stream(B):
        assert big.enqueue() == api.CLOSURE_RESIDENT
        assert big.right()
