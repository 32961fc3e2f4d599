"""The two-launch batched pack (four lanes per block, tiles of 32 blocks, eight
per warp) against the oracle, byte for byte: block counts around the edges
of a warp's and a CTA's share and over groups of 32 and 1024 tiles, streams and whole
batches that start at any word, partial blocks, and every shape of block."""
import numpy as np
import pytest

import oracle_ref as O
from gen import KINDS32, KINDS64, streams

pytestmark = pytest.mark.gpu

# values per stream: 1..33 blocks, partial ends, empty streams between
TABLES = {
    "one_value": [1],
    "warp_edge": [8 * 128 - 1, 0, 0, 129],
    "tile_edge": [31 * 128, 128, 1],
    "ragged": [1, 2, 3, 127, 128, 130, 0, 1003, 5, 4096, 77, 261],
    "many_short": [7] * 200 + [0] * 50 + [129] * 40,
}


@pytest.fixture(scope="module")
def env():
    import torch

    import utlpfor_b200 as U
    from utlpfor_b200._lib import load
    L = load()
    old = L.utl_get_knob(2)
    assert L.utl_set_knob(2, 3) == 0
    yield U, torch
    L.utl_set_knob(2, old)


def _check(U, torch, vals, vo, flag, skew=0):
    want, wbo, wso = O.pack_streams(flag, vals, vo)
    it = vals.dtype.itemsize
    host = np.zeros(len(vals) + skew, vals.dtype)
    host[skew:] = vals
    d = torch.from_numpy(host.view(np.int64 if it == 8 else np.int32)).cuda()[skew:]
    pb = U.pack_batch(d, vo, flag)
    assert pb.packed_len == len(want)
    assert np.array_equal(pb.packed[:len(want)].cpu().numpy(), want)
    assert np.array_equal(pb.block_off.cpu().numpy().view(np.uint64), wbo)
    assert np.array_equal(pb.stream_byte_off.cpu().numpy().view(np.uint64), wso)


@pytest.mark.parametrize("flag", [0, 1, 2, 3, 4, 5, 6, 7, 8, 16 | 1])
@pytest.mark.parametrize("kind", KINDS32)
@pytest.mark.parametrize("table", sorted(TABLES))
def test_u32(env, table, kind, flag):
    U, torch = env
    vals, vo = streams(np.random.default_rng(7 * flag + len(kind)), TABLES[table], kind)
    _check(U, torch, vals, vo, flag, skew=flag % 4)


@pytest.mark.parametrize("flag", [0, 1, 2, 3, 4, 5, 8 | 1])
@pytest.mark.parametrize("kind", KINDS64)
@pytest.mark.parametrize("table", sorted(TABLES))
def test_u64(env, table, kind, flag):
    U, torch = env
    vals, vo = streams(np.random.default_rng(9 * flag + len(kind)), TABLES[table], kind, is64=True)
    _check(U, torch, vals, vo, flag, skew=flag % 2)


@pytest.mark.parametrize("is64", [False, True])
def test_u64_minimum_across_high_words(env, is64):
    """Blocks whose high words differ by one: FOR64 exactly when max - min
    stays below 2^32; and the same batch as uint32 values."""
    U, torch = env
    rng = np.random.default_rng(3)
    v = np.uint64(2**33 - 1000) + rng.integers(0, 2000, 128 * 40, dtype=np.uint64)
    v[5 * 128 + 3] = 2**33 - 1000 + 2**32 - 1  # still fits
    v[5 * 128 + 9] = 2**33 - 1000
    v[9 * 128 + 3] = 2**33 - 1000 + 2**32      # one too far
    v[9 * 128 + 9] = 2**33 - 1000
    v = v if is64 else (v & np.uint64(0xFFFFFFFF)).astype(np.uint32)
    for flag in (0, 1, 2):
        _check(U, torch, v, np.array([0, len(v)], np.uint64), flag)


@pytest.mark.parametrize("is64", [False, True])
@pytest.mark.parametrize("flag", [0, 1, 4])
def test_many_tiles(env, is64, flag):
    """Offsets over whole groups of tiles; streams end anywhere."""
    U, torch = env
    rng = np.random.default_rng(11 + flag)
    lens = [700003, 1, 128 * 32 * 70, 1500001 if is64 else 4500001, 0, 333]
    kinds = KINDS64 if is64 else ("exc", "sorted", "dense_exc", "wide")
    parts = [streams(rng, [n], kinds[i % len(kinds)], is64=is64)[0] for i, n in enumerate(lens)]
    vo = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    _check(U, torch, np.concatenate(parts), vo, flag, skew=1)


def test_capacity_is_reported(env):
    U, torch = env
    v = torch.arange(128 * 100, dtype=torch.int32, device="cuda")
    codec = U.BatchCodec(np.array([0, v.numel()], np.uint64), flag=0, out_cap=3000)
    codec.packed.fill_(7)
    codec.pack(v)
    torch.cuda.synchronize()
    assert codec.error_bits() & (1 << 9)
    U.BatchCodec(np.array([0, v.numel()], np.uint64), flag=0).pack(v)
