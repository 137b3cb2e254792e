"""NMH builds around the sort's tile edges and the tile count from which the
sort takes a scan launch, with many equal keys (stability of the sort)."""
import numpy as np
import pytest

from aurora_gb300 import api, scenes
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("equal", [False, True])
@pytest.mark.parametrize("n", [2048, 2050, 6143, 63487, 65534, 65535, 65536, 65537, 67584, 67586])
def test_build_equals_the_oracle_at_sort_tile_edges(n, equal):
    import torch
    V = scenes.random_soup(n, seed=n)
    if equal:
        V = np.round(V * np.float32(8.0)).astype(np.float32)
    ctx = api.Context(0)
    nmh = api.Nmh(ctx, torch.from_numpy(np.ascontiguousarray(V).reshape(-1)).cuda(), count=n)
    perm, _ = nmh.export()
    operm, olv = oracle.nmh_build(V)
    assert nmh.info()[1] == olv
    assert np.array_equal(perm, operm)
