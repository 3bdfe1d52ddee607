"""How a stream is cut into groups of batches (orca_group_sizes): every batch once, no group above the limit."""
import numpy as np
import pytest

from orca_b200 import _lib, build


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("bs,k", [(1, 1), (37, 10), (200, 10), (600, 20), (1000, 10), (2000, 10), (30000, 20)])
def test_groups_cover_the_stream(mode, bs, k):
    build.build()
    L = _lib.lib()
    most = L.orca_group_size(bs, k, 2, mode)
    assert 1 <= most <= 32
    for n in [*range(1, 200), 3917]:
        sizes = np.full(n, -7, dtype=np.int32)
        g = L.orca_group_sizes(n, bs, k, 2, mode, sizes.ctypes.data)
        s = sizes[:g]
        assert s.sum() == n and s.min() >= 1 and s.max() <= most
