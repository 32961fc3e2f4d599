"""Batched Get position by position against the oracle's Get: position-list
and bitmap exceptions with and without delta, partial blocks, packed buffers
that start at any byte, and damaged blocks (which the direct path has to
leave to the checked one or answer as the reference does)."""
import ctypes as C

import numpy as np
import pytest

import oracle_ref as O
from gen import streams

pytestmark = pytest.mark.gpu

LENS = [128 * 3, 1, 77, 129, 16, 0, 300]


def _p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("damage", [False, True])
@pytest.mark.parametrize("flag", [0, 1, 2, 3, 5])
@pytest.mark.parametrize("kind,is64", [("exc", False), ("dense_exc", False), ("sorted", False), ("walk", False),
                                       ("wide", False), ("for64", True), ("full", True), ("walk", True),
                                       ("upper_for", True)])
def test_every_position(kind, is64, flag, damage):
    import torch

    from utlpfor_b200._lib import load
    L = load()
    rng = np.random.default_rng(50 + flag)
    vals, vo = streams(rng, LENS, kind, is64=is64)
    packed, bo, _ = O.pack_streams(flag, vals, vo)
    if damage:
        packed = packed.copy()
        for b in range(len(bo) - 1):
            for at in rng.integers(int(bo[b]), int(bo[b + 1]), 2):
                packed[at] ^= 1 << int(rng.integers(0, 8))
    skew = flag % 4
    buf = torch.zeros(len(packed) + skew, dtype=torch.uint8, device="cuda")
    buf[skew:] = torch.from_numpy(packed)
    d_p = buf[skew:]
    d_bo = torch.from_numpy(bo.view(np.int64)).cuda()
    d_vo = torch.from_numpy(vo.view(np.int64)).cuda()
    bs = torch.empty(len(vo), dtype=torch.int64, device="cuda")
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.utl_batch_plan(_p(d_vo), len(LENS), _p(bs), st) == 0
    qs = np.repeat(np.arange(len(LENS)), LENS).astype(np.uint32)
    qp = np.concatenate([np.arange(n) for n in LENS]).astype(np.uint64)
    d_qs, d_qp = torch.from_numpy(qs.view(np.int32)).cuda(), torch.from_numpy(qp.view(np.int64)).cuda()
    out = torch.zeros(len(qs), dtype=torch.int64 if is64 else torch.int32, device="cuda")
    status = torch.zeros(len(qs), dtype=torch.int32, device="cuda")
    fn = L.utl_get_batch_u64 if is64 else L.utl_get_batch_u32
    assert fn(_p(d_p), len(packed), _p(d_bo), _p(d_vo), _p(bs), len(LENS), _p(d_qs), _p(d_qp), len(qs), _p(out),
              _p(status), None, st) == 0
    out, status = out.cpu().numpy().view(vals.dtype), status.cpu().numpy()
    starts = bs.cpu().numpy()
    for i in range(len(qs)):
        b = int(starts[qs[i]]) + int(qp[i]) // 128
        v, err, ovf = (O.get_u64 if is64 else O.get_u32)(int(qp[i]) % 128, packed[int(bo[b]):int(bo[b + 1])])
        assert (status[i] & 0xFF, status[i] >> 8) == (err, ovf), i
        if err == 0:
            assert out[i] == v, i
        if not damage and kind != "upper_for":
            assert err == 0 and out[i] == vals[int(vo[qs[i]]) + int(qp[i])], i
