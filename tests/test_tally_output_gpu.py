"""How the count's tiles go out: whole and cut, inside the matrix and at its edge, into rows that are aligned to 16
bytes and others, overwriting and adding, against the oracle."""
import numpy as np
import pytest
import torch

from scalingelections_b200 import _lib, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 40, 3001])  # three: whole tiles, and some of them cut
@pytest.mark.parametrize("C", [127, 128, 129, 256, 300, 384])
def test_output(orc, C, V):
    rng = np.random.default_rng(C * 10 + V)
    rows = np.stack([rng.permutation(C) for _ in range(V)]).astype(np.int32)
    want = orc.tally(rows, "positions").astype(np.int64)
    ids = torch.from_numpy(rows.reshape(-1)).cuda()
    w = torch.empty(api.tally_workspace_bytes(V, C), dtype=torch.uint8, device="cuda")
    for ld, shift in ((C, 0), (-(-C // 4) * 4, 0), (-(-C // 4) * 4 + 1, 0), (-(-C // 4) * 4, 1)):
        flat = torch.full((C * ld + shift,), 5, dtype=torch.int32, device="cuda")
        out = flat[shift:].view(C, ld)
        keep = out[:, C:].clone()
        for flags, start in ((0, 0), (1, want)):  # overwrite, then add the same ballots again
            _lib.check(_lib.lib().se_tally_ex(ids.data_ptr(), 4, None, 0, V, C, flags, out.data_ptr(), ld, w.data_ptr(),
                                              w.numel(), torch.cuda.current_stream().cuda_stream))
            assert np.array_equal(out[:, :C].cpu().numpy(), want + start), (ld, shift, flags)
        assert torch.equal(out[:, C:], keep)
