"""Per-call decode: packed input staged in whole 16-byte pieces, two a lane.
Blocks of every width with tails that move the staged length around the
pieces' and the rounds' ends (16, 512, 1024 bytes), each after a longer one
whose bytes are still in the staging area; truncated input gives the
oracle's status."""
import numpy as np
import pytest

import oracle_ref as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def U():
    import utlpfor_b200 as U
    return U


def code_of(U, fn):
    try:
        return fn(), 0
    except U.UTLError as e:
        return None, e.code


@pytest.mark.parametrize("is64", [False, True], ids=["u32", "u64"])
@pytest.mark.parametrize("width", [0, 4, 8, 16, 24, 28, 32])
def test_pieces(U, is64, width):
    rng = np.random.default_rng(width + 100 * is64)
    top = (1 << width) - 1
    v = rng.integers(0, top, 128, dtype=np.uint32, endpoint=True).astype(np.uint32)
    full = rng.integers(0, 1 << 32, 128, dtype=np.uint64).astype(np.uint32)
    if is64:
        v = v.astype(np.uint64) | (rng.integers(0, top, 128, dtype=np.uint64, endpoint=True) << np.uint64(32))
        full = full.astype(np.uint64) | (full.astype(np.uint64) << np.uint64(32))
    pack, unpack, get = (O.pack_u64, O.unpack_u64, O.get_u64) if is64 else (O.pack_u32, O.unpack_u32, O.get_u32)
    up, gt = (U.UnpackUint64, U.GetUint64) if is64 else (U.UnpackUint32, U.GetUint32)
    flag = U.NoPatch | U.NoFOR
    long, block = bytes(pack(flag, full)[0]), bytes(pack(flag, v)[0])
    for tail in (0, 1, 11, 12, 13, 27, 28, 29, 64, 65, 600):
        up(long)
        got, used = up(block + b"\xa5" * tail)
        assert used == len(block) and np.array_equal(np.asarray(got, dtype=v.dtype), v)
        up(long)
        assert gt(127, block + b"\xa5" * tail) == int(v[127])
    for cut in (1, 5, 15, 16, 17, len(block) - 16, len(block) - 1):
        if 0 < cut < len(block):
            up(long)
            assert code_of(U, lambda: up(block[:cut]))[1] == unpack(block[:cut])[2]
            assert code_of(U, lambda: gt(127, block[:cut]))[1] == get(127, block[:cut])[1]
