"""Batched Get of blocks at the ends of the packed buffer: buffers that start and
end at any byte of a word, of one block and of a few, queried in any order, with
bytes around the buffer that would show if they were used; and damaged ends."""
import ctypes as C

import numpy as np
import pytest

import oracle_ref as O
from gen import streams

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("damage", [False, True])
@pytest.mark.parametrize("n", [1, 128, 200, 128 * 3 + 5])
@pytest.mark.parametrize("kind,is64,flag", [("exc", False, 0), ("exc", False, 1), ("dense_exc", False, 1),
                                            ("sorted", False, 1), ("wide", False, 4), ("for64", True, 0),
                                            ("walk", True, 1), ("upper_for", True, 0)])
def test_every_alignment_of_both_ends(kind, is64, flag, n, damage):
    import torch

    from utlpfor_b200._lib import load
    L = load()
    fn = L.utl_get_batch_u64 if is64 else L.utl_get_batch_u32
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    rng = np.random.default_rng(n + flag)
    ends = set()
    for seed in range(12):  # lengths of the packed buffer of every remainder, where the data has them
        vals, vo = streams(np.random.default_rng(seed), [n], kind, is64=is64)
        packed, bo, _ = O.pack_streams(flag, vals, vo)
        if len(packed) % 4 in ends:
            continue
        ends.add(len(packed) % 4)
        packed = packed.copy()
        if damage:
            for b in (0, len(bo) - 2):
                for at in rng.integers(int(bo[b]), int(bo[b + 1]), 2):
                    packed[at] ^= 1 << int(rng.integers(0, 8))
        d_bo = torch.from_numpy(bo.view(np.int64)).cuda()
        d_vo = torch.from_numpy(vo.view(np.int64)).cuda()
        d_bs = torch.tensor([0, len(bo) - 1], dtype=torch.int64, device="cuda")
        qp = rng.integers(0, n, 700)
        d_qs = torch.zeros(len(qp), dtype=torch.int32, device="cuda")
        d_qp = torch.from_numpy(qp).cuda()
        want = []
        for pos in range(n):
            b = pos // 128
            want.append((O.get_u64 if is64 else O.get_u32)(pos % 128, packed[int(bo[b]):int(bo[b + 1])]))
        for skew in range(4):
            buf = torch.full((len(packed) + 8,), 0xFF, dtype=torch.uint8, device="cuda")
            d = buf[skew:skew + len(packed)]
            d.copy_(torch.from_numpy(packed))
            out = torch.zeros(len(qp), dtype=torch.int64 if is64 else torch.int32, device="cuda")
            status = torch.zeros(len(qp), dtype=torch.int32, device="cuda")
            assert fn(_p(d), len(packed), _p(d_bo), _p(d_vo), _p(d_bs), 1, _p(d_qs), _p(d_qp), len(qp), _p(out),
                      _p(status), None, st) == 0
            got, stat = out.cpu().numpy().view(vals.dtype), status.cpu().numpy()
            for i, pos in enumerate(qp):
                v, err, ovf = want[int(pos)]
                assert (stat[i] & 0xFF, stat[i] >> 8) == (err, ovf), (skew, pos)
                if err == 0:
                    assert got[i] == v, (skew, pos)
                if not damage and kind != "upper_for":  # the reference misreads its upper halves' 4-byte base
                    assert err == 0 and got[i] == vals[int(pos)], (skew, pos)
