"""The stream indexer on blocks far longer than any a packer writes, which
BlockLength accepts (the StreamVByte length is 16 bits, block_length.go:41-48):
they span whole partitions and regions, and their bytes parse as a chain of
blocks of their own."""
import numpy as np
import pytest

import oracle_ref as O
from gen import streams

pytestmark = pytest.mark.gpu


def long_block(svb, fill):
    """count 128, width 0, uint32, one exception, svb bytes of StreamVByte data."""
    head = np.array([0x0100_4080], dtype="<u4").view(np.uint8)
    body = np.resize(fill, svb)
    return np.concatenate([head, np.array([svb & 255, svb >> 8, 5], np.uint8), body])


@pytest.mark.parametrize("svb", [9000, 20001, 40002, 65535])
@pytest.mark.parametrize("fill", ["headers", "zeros"])
def test_offsets(fill, svb):
    import torch

    import utlpfor_b200 as U
    rng = np.random.default_rng(svb)
    # 4-byte blocks: count 1, width 0, uint32
    bytes_of = {"headers": np.array([0x00004001], "<u4").view(np.uint8), "zeros": np.zeros(4, np.uint8)}[fill]
    parts = []
    for i in range(9):
        vals, vo = streams(rng, [int(rng.integers(1, 30000))], ("exc", "sorted", "full")[i % 3])
        parts += [O.pack_streams(0, vals, vo)[0], long_block(svb, bytes_of), long_block(int(rng.integers(1, svb)), bytes_of)]
    p = np.concatenate(parts)
    want, err, _ = O.index_stream(p)
    assert err == O.OK
    got = U.index_stream(torch.from_numpy(p).cuda()).cpu().numpy()
    assert np.array_equal(got, np.array(want, np.int64))
    # and with a bad block behind them
    bad = np.concatenate([p, np.array([200, 0, 0, 0], np.uint8), p])
    _, err, at = O.index_stream(bad)
    with pytest.raises(Exception) as e:
        U.index_stream(torch.from_numpy(bad).cuda())
    assert e.value.code == err and e.value.block == at
