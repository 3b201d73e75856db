"""The variant table decides whether the automatic schedule runs the one-launch closure in registers: a table of
the caller's own that does not name it is followed at every size."""
import numpy as np
import pytest
import torch

from scalingelections_b200 import LANES_U16, LANES_U32, api, autotune


@pytest.fixture(autouse=True)
def builtin_table():
    yield
    api.set_closure_variants(api.BUILTIN_CLOSURE_VARIANTS)


def form(C, lanes=LANES_U16):
    return api.CLOSURE_RESIDENT if api.closure_is_resident(C, lanes) else api.closure_schedule(C, lanes)


def test_own_table():
    api.set_closure_variants([(600, 3), (2048, 7)])
    assert [form(C) for C in (1, 600, 601, 1536, 2049)] == [3, 3, 7, 7, 1]
    api.set_closure_variants([])
    assert [form(C) for C in (1, 1536)] == [1, 1]
    api.set_closure_variants([(600, 9), (4096, 8)])
    assert [form(C) for C in (600, 601, 1536)] == [9, 8, 8]
    api.set_closure_variants([(600, 4), (2048, 9), (4096, 8)])  # passed over where it does not fit
    assert [form(C) for C in (600, 601, 1536, 1537, 2048)] == [4, 9, 9, 8, 8]
    assert [form(C, LANES_U32) for C in (1344, 1345)] == [9, 6]


def test_builtin_table():
    for _ in range(2):
        assert [form(C) for C in (1, 1024, 1536, 1537, 4096, 4097)] == [9, 9, 9, 8, 8, 6]
        assert [form(C, LANES_U32) for C in (1344, 1345)] == [9, 6]
        api.set_closure_variants(api.BUILTIN_CLOSURE_VARIANTS)


@pytest.mark.parametrize("mode", [-1, 0, 2, 10])
def test_refused_modes(mode):
    with pytest.raises(api.SchulzeError, match="table modes"):
        api.set_closure_variants([(600, mode)])
    assert form(600) == api.CLOSURE_RESIDENT


@pytest.mark.gpu
def test_own_table_runs():
    d = api._to_device_u32(np.random.default_rng(1).integers(0, 9000, size=(520, 520)).astype(np.uint32), "cuda")
    want = api.strongest_paths_device(d, lanes=LANES_U16).view(torch.int32)
    assert api.last_closure_schedule() == api.CLOSURE_RESIDENT
    for table, ran in (([(600, 3)], 3), ([(600, 9)], 9), ([(500, 9)], 1), ([], 1)):
        api.set_closure_variants(table)
        assert torch.equal(api.strongest_paths_device(d, lanes=LANES_U16).view(torch.int32), want)
        assert api.last_closure_schedule() == ran, table


@pytest.mark.gpu
def test_tuner_times_the_form_that_runs():
    api.set_closure_variants([(700, 4)])
    res = autotune.tune_closure([640, 1600], reps=1, install=False)
    assert api.CLOSURE_RESIDENT in res["sizes"][640] and api.CLOSURE_RESIDENT not in res["sizes"][1600]
    assert form(640) == 4  # the caller's table is back
    autotune.tune_closure([640], reps=1)
    assert form(640) in autotune.CLOSURE_MODES
