"""The default uint32 unpack on both sides of the batch size at which it goes
from four lanes per block to a thread per block (22732 blocks on 148 SMs),
against the packed values, in ragged streams."""
import numpy as np
import pytest

from gen import streams

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flag", [0, 1])
@pytest.mark.parametrize("kind", ["exc", "sorted", "walk", "const"])
@pytest.mark.parametrize("blocks", [22732, 22733])
def test_round_trip(blocks, kind, flag):
    import torch

    import utlpfor_b200 as U
    lens = [128 * 50 - 3] * 300 + [1, 127]
    lens.append(128 * (blocks - sum((n + 127) // 128 for n in lens)) - 5)
    vals, vo = streams(np.random.default_rng(blocks + flag), lens, kind)
    d = torch.from_numpy(vals.view(np.int32)).cuda()
    pb = U.pack_batch(d, vo, flag)
    assert pb.n_blocks == blocks
    assert torch.equal(U.unpack_batch(pb), d)
