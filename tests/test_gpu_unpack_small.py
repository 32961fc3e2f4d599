"""The default uint32 unpack on both sides of the batch size up to which it
decodes four lanes per block (37888 blocks), against the packed values:
list exceptions, bitmaps, delta, partial blocks and streams at any word."""
import numpy as np
import pytest

from gen import streams

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flag", [0, 1, 4])
@pytest.mark.parametrize("kind", ["exc", "dense_exc", "sorted", "walk"])
@pytest.mark.parametrize("blocks", [1, 8, 9, 37888, 37889])
def test_round_trip(blocks, kind, flag):
    import torch

    import utlpfor_b200 as U
    head = min(5, blocks - 1)  # short streams first: the long one starts at an odd word
    lens = [1, 127, 3, 64, 17][:head] + [128 * (blocks - head) - 5]
    vals, vo = streams(np.random.default_rng(blocks + flag), lens, kind)
    d = torch.from_numpy(vals.view(np.int32)).cuda()
    pb = U.pack_batch(d, vo, flag)
    assert pb.n_blocks == blocks
    out = U.unpack_batch(pb)
    assert torch.equal(out, d)
