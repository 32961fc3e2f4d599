"""The stream indexer with its waits cut short (UTL_KNOB_SPIN_LIMIT): a region
whose staged bytes or whose entry do not come in time gives up, and the call
must still return the oracle's offsets; and it does again at the default."""
import numpy as np
import pytest

import oracle_ref as O
from gen import streams

pytestmark = pytest.mark.gpu

SPIN_LIMIT = 4


@pytest.mark.parametrize("skew", [0, 5])
@pytest.mark.parametrize("n", [100, 128 * 40, 128 * 9000 + 3])
@pytest.mark.parametrize("limit", [1, 2])
def test_short_waits(limit, n, skew):
    import torch

    import utlpfor_b200 as U
    from utlpfor_b200._lib import load
    L = load()
    vals, vo = streams(np.random.default_rng(n + limit), [n], "exc")
    packed, bo, _ = O.pack_streams(0, vals, vo)
    buf = torch.zeros(len(packed) + 16, dtype=torch.uint8, device="cuda")
    d = buf[skew:skew + len(packed)]
    d.copy_(torch.from_numpy(packed))
    want = bo.astype(np.int64)
    old = L.utl_get_knob(SPIN_LIMIT)
    try:
        assert L.utl_set_knob(SPIN_LIMIT, limit) == 0
        for _ in range(3):
            assert np.array_equal(U.index_stream(d).cpu().numpy(), want)
    finally:
        L.utl_set_knob(SPIN_LIMIT, old)
    assert np.array_equal(U.index_stream(d).cpu().numpy(), want)
