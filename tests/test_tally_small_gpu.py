"""The tally of few candidates or voters, whose tiles are cut into many voter ranges, against the
oracle, and the check of the ballot index that the tally makes as it reads it."""
import numpy as np
import pytest
import torch

from scalingelections_b200 import api

pytestmark = pytest.mark.gpu


def ballots(V, C, ragged, seed):
    rng = np.random.default_rng(seed)
    rows = [rng.permutation(C).astype(np.int32) for _ in range(V)]
    if ragged:
        rows = [r[:rng.integers(1, C + 1)] for r in rows]
    return rows


def to_device(rows):
    offs = np.zeros(len(rows) + 1, dtype=np.int64)
    np.cumsum([len(r) for r in rows], out=offs[1:])
    return torch.from_numpy(np.concatenate(rows)).cuda(), torch.from_numpy(offs).cuda()


def completed(rows, C):
    return np.stack([np.concatenate([r, np.setdiff1d(np.arange(C, dtype=np.int32), r)]) for r in rows]).astype(np.int32)


@pytest.mark.parametrize("V", [1, 63, 64, 65, 129, 2000])
@pytest.mark.parametrize("C", [1, 3, 128, 129, 300])
@pytest.mark.parametrize("ragged", [False, True])
def test_few_tiles(orc, V, C, ragged):
    rows = ballots(V, C, ragged, seed=V * 1000 + C)
    ids, offs = to_device(rows)
    got = api._to_host_u32(api.tally_device(ids, offs, C))
    assert np.array_equal(got, orc.tally(completed(rows, C), "positions"))


@pytest.mark.parametrize("V", [31, 65, 290])
@pytest.mark.parametrize("C", [1000, 2300, 2433])
def test_whole_rounds_and_cut_tiles(orc, V, C):
    """36 tiles, all cut; 171 and 190 above the diagonal, a round of whole tiles on 148 SMs and the
    rest whole (few voters) or cut (many); ballots that repeat a candidate in whole and cut tiles."""
    rows = ballots(V, C, False, seed=V + C)
    ids, offs = to_device(rows)
    got = api._to_host_u32(api.tally_device(ids, offs, C))
    assert np.array_equal(got, orc.tally(np.stack(rows), "positions"))
    for v in (0, V // 2, V - 1):
        rows[v][1] = rows[v][0]
    ids, offs = to_device(rows)
    got = api._to_host_u32(api.tally_device(ids, offs, C))
    assert np.array_equal(got, orc.tally(np.stack(rows), "scatter"))


@pytest.mark.parametrize("C", [40, 2050])
def test_bad_offsets_are_refused(C):
    rows = ballots(70, C, False, seed=C)
    ids, offs = to_device(rows)
    good = api.tally_device(ids, offs, C).view(torch.int32)
    for at, value in ((0, 1), (0, -5), (70, 70 * C - 1), (70, 70 * C + 1), (70, 1 << 40), (33, 34 * C + 1),
                      (33, -1), (33, 1 << 50)):
        bad = offs.clone()
        bad[at] = value
        with pytest.raises(ValueError, match="offsets must start at 0"):
            api.tally_device(ids, bad, C)
    assert torch.equal(api.tally_device(ids, offs, C).view(torch.int32), good)
    bad_id = ids.clone()
    bad_id[5] = C
    with pytest.raises(api.SchulzeError, match="outside"):
        api.tally_device(bad_id, offs, C)
