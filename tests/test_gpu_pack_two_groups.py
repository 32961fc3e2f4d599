"""The two-launch pack beyond the sizes of test_gpu_pack_two.py, through the C
ABI: batches of more than 1024 tiles of 32 blocks, whose offsets go over groups
of tiles that have to start at zero in a scratch full of something else; what it
leaves alone when the output is too small; and every flag."""
import ctypes as C

import numpy as np
import pytest

import oracle_ref as O
from gen import KINDS32, KINDS64, streams

pytestmark = pytest.mark.gpu

PACK_SCHEDULE = 2
CAPACITY_BIT = 1 << 9


def _p(t):
    return C.c_void_p(t.data_ptr())


class Batch:
    """A batch on the device; pack() gives error bits, packed bytes, offsets and
    the bytes after the capacity the pack was told, every buffer filled before."""

    def __init__(self, torch, L, vals, vo, flag, skew=0):
        self.torch, self.L, self.flag = torch, L, flag
        self.is64 = vals.dtype.itemsize == 8
        host = np.zeros(len(vals) + skew, vals.dtype)
        host[skew:] = vals
        self.vals = torch.from_numpy(host.view(np.int64 if self.is64 else np.int32)).cuda()[skew:]
        self.vo = torch.from_numpy(vo.view(np.int64)).cuda()
        self.ns = len(vo) - 1
        self.bs = torch.empty(self.ns + 1, dtype=torch.int64, device="cuda")
        assert L.utl_batch_plan(_p(self.vo), self.ns, _p(self.bs), None) == 0
        self.nb = L.utl_count_blocks(vo.ctypes.data_as(C.POINTER(C.c_uint64)), self.ns)

    def pack(self, cap=None):
        torch, L = self.torch, self.L
        per = L.utl_max_block_length64(self.flag) if self.is64 else L.utl_max_block_length32(self.flag)
        size = self.nb * per
        cap = size if cap is None else cap
        out = torch.full((size + 64,), 7, dtype=torch.uint8, device="cuda")
        bo = torch.full((self.nb + 1,), -1, dtype=torch.int64, device="cuda")
        sb = L.utl_pack_scratch_bytes(self.nb)
        scratch = torch.full((sb + 64,), 0xA5, dtype=torch.uint8, device="cuda")
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        n0 = L.utl_launch_count()
        fn = L.utl_pack_batch_u64 if self.is64 else L.utl_pack_batch_u32
        assert fn(self.flag, _p(self.vals), _p(self.vo), _p(self.bs), self.ns, self.nb, _p(out), cap, _p(bo), None,
                  _p(scratch), sb, _p(err), None) == 0
        torch.cuda.synchronize()
        assert bool((scratch[sb:] == 0xA5).all())
        self.launches = L.utl_launch_count() - n0
        return int(err.item()), out.cpu().numpy(), bo.cpu().numpy().view(np.uint64), cap


@pytest.fixture(scope="module")
def env():
    import torch

    from utlpfor_b200._lib import load
    L = load()
    old = L.utl_get_knob(PACK_SCHEDULE)
    assert L.utl_set_knob(PACK_SCHEDULE, 3) == 0
    yield torch, L
    L.utl_set_knob(PACK_SCHEDULE, old)


def _check(b, vals, vo):
    want, wbo, _ = O.pack_streams(b.flag, vals, vo, n_threads=8)
    err, out, bo, _ = b.pack()
    assert err == 0 and b.launches == 2
    assert np.array_equal(bo, wbo)
    assert np.array_equal(out[:len(want)], want)
    assert bool((out[len(want):] == 7).all())


@pytest.mark.parametrize("flag", [0, 1])
def test_u64_groups(env, flag):
    torch, L = env
    rng = np.random.default_rng(21 + flag)
    lens = [900001, 3, 128 * 32 * 1024 + 128 * 31, 0, 77, 128 * 40]
    kinds = ("for64", "full", "walk", "zero", "fit32", "walk")
    vals = np.concatenate([streams(rng, [n], k, is64=True)[0] for n, k in zip(lens, kinds)])
    vo = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    b = Batch(torch, L, vals, vo, flag, skew=1)
    assert b.nb > 1024 * 32
    _check(b, vals, vo)


@pytest.mark.parametrize("flag", [4, 5])
def test_u32_nopatch_groups(env, flag):
    torch, L = env
    rng = np.random.default_rng(31 + flag)
    lens = [700003, 1, 128 * 32 * 1024, 333]
    vals = np.concatenate([streams(rng, [n], k)[0] for n, k in zip(lens, ("exc", "wide", "full", "dense_exc"))])
    vo = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    b = Batch(torch, L, vals, vo, flag, skew=3)
    assert b.nb > 1024 * 32
    b.pack()  # large blocks: from now on such batches take the two launches
    _check(b, vals, vo)


@pytest.mark.parametrize("is64", [False, True])
@pytest.mark.parametrize("blocks", [1, 100])
def test_too_small_an_output(env, blocks, is64):
    """The error is reported, the offsets are those of the whole batch, and not
    a byte past the capacity is written; the next pack is right."""
    torch, L = env
    vals, vo = streams(np.random.default_rng(blocks), [128 * blocks - 9], "full", is64=is64)
    b = Batch(torch, L, vals, vo, 0)
    want, wbo, _ = O.pack_streams(0, vals, vo)
    for cap in (0, 1, len(want) // 2, len(want) - 1):
        err, out, bo, _ = b.pack(cap)
        assert err == CAPACITY_BIT
        assert np.array_equal(bo, wbo)
        assert bool((out[cap:] == 7).all()), cap
    _check(b, vals, vo)


@pytest.mark.parametrize("flag", list(range(16)) + [16 | 5, 32 | 9, 48 | 15])
@pytest.mark.parametrize("is64", [False, True])
def test_every_flag(env, is64, flag):
    torch, L = env
    rng = np.random.default_rng(400 + flag)
    for kind in (KINDS64 if is64 else KINDS32):
        vals, vo = streams(rng, [300, 1, 0, 129, 128 * 9, 64], kind, is64=is64)
        _check(Batch(torch, L, vals, vo, flag, skew=flag % 2), vals, vo)
