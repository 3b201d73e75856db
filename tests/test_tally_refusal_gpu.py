"""A bad ballot index is refused as it was when it was checked before the tally: a ValueError, whatever the
ids, and the caller's output as it was."""
import numpy as np
import pytest
import torch

from scalingelections_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [40, 700, 2050])
def test_bad_offsets_leave_the_output_alone(C):
    V = 70
    rows = np.stack([np.random.default_rng(v).permutation(C) for v in range(V)]).astype(np.int32)
    rows[5, 1] = rows[5, 0]  # a repeat: counted by its own kernel
    ids = torch.from_numpy(rows.reshape(-1)).cuda()
    offs = torch.arange(V + 1, dtype=torch.int64, device="cuda") * C
    big = torch.full((C, C + 3), 7, dtype=torch.int32, device="cuda")
    for at, value in ((0, 1), (33, 34 * C + 1), (V, V * C - 1)):
        bad = offs.clone()
        bad[at] = value
        with pytest.raises(ValueError, match="offsets must start at 0"):
            api.tally_device(ids, bad, C, out=big.view(torch.uint32)[:, :C])
        assert bool((big == 7).all()), (at, value)
    api.tally_device(ids, offs, C, out=big.view(torch.uint32)[:, :C])
    assert torch.equal(big[:, :C], api.tally_device(ids, offs, C).view(torch.int32))
    assert bool((big[:, C:] == 7).all())


def test_bad_offsets_without_ids():
    ids = torch.empty(0, dtype=torch.int32, device="cuda")
    with pytest.raises(ValueError, match="offsets must start at 0"):
        api.tally_device(ids, torch.tensor([0, 2, 4], device="cuda"), 4)
