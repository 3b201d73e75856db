"""Strongest paths that run the length of the matrix through the one-launch closure's shapes of more than one block
per CTA (16-bit lanes from C = 1089 on, two; 32-bit lanes likewise, three), ragged last tiles among them, against
the oracle."""
import numpy as np
import pytest

from conftest import chain_forward_ok, chain_matrix
from scalingelections_b200 import LANES_AUTO, LANES_U16, LANES_U32, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [1089, 1217, 1344, 1409, 1536])
@pytest.mark.parametrize("order", ["shuffled", "ascending", "descending"])
def test_chain(orc, C, order):
    P, perm, w = chain_matrix(C, seed=C, order=order)
    S_ref = orc.strongest_paths(P, "blocked", tile=16)
    assert chain_forward_ok(S_ref, perm, w)
    d = api._to_device_u32(np.ascontiguousarray(P, dtype=np.uint32), "cuda")
    for lanes in (LANES_U16, LANES_AUTO) + ((LANES_U32,) if C <= 1344 else ()):
        S = api._to_host_u32(api.strongest_paths_device(d, lanes=lanes))
        assert api.last_closure_schedule() == api.CLOSURE_RESIDENT
        assert np.array_equal(S, S_ref), lanes
