"""The stream indexer's regions (32256 bytes, teams of 1008) against the
oracle's BlockLength walk: streams that end around region and team edges,
start at any byte, and whose blocks are far smaller or larger than a team's
bytes."""
import numpy as np
import pytest

import oracle_ref as O
from gen import streams

pytestmark = pytest.mark.gpu

REGION, TEAM = 32256, 1008


def packed_of(kind, n, flag, is64):
    vals, vo = streams(np.random.default_rng(n + flag), [n], kind, is64=is64)
    return O.pack_streams(flag, vals, vo)[0]


@pytest.mark.parametrize("skew", [0, 1, 7, 15])
@pytest.mark.parametrize("kind,flag,is64", [("exc", 0, False), ("exc", 2, False), ("zero", 0, False),
                                            ("full", 4, False), ("full", 0, True), ("for64", 1, True)])
def test_edges(kind, flag, is64, skew):
    import torch

    import utlpfor_b200 as U
    whole = packed_of(kind, 128 * (260 if kind != "zero" else 17000), flag, is64)
    bo, err, _ = O.index_stream(whole)
    assert err == O.OK
    bo = np.array(bo)
    ends = set()
    for edge in (16, TEAM, REGION - TEAM, REGION, REGION + 16, 2 * REGION, len(whole)):
        i = int(np.searchsorted(bo, edge))
        ends.update(int(bo[k]) for k in (i - 1, i, i + 1) if 0 < k < len(bo))
    buf = torch.zeros(len(whole) + 64, dtype=torch.uint8, device="cuda")
    for e in sorted(ends):
        buf[skew:skew + e] = torch.from_numpy(whole[:e].copy()).cuda()
        got = U.index_stream(buf[skew:skew + e]).cpu().numpy()
        assert np.array_equal(got, bo[bo <= e]), e


def test_capacity():
    import ctypes as C

    import torch

    from utlpfor_b200._lib import load
    L = load()
    p = packed_of("exc", 128 * 700, 0, False)
    d = torch.from_numpy(p).cuda()
    for cap, rc in ((700, 0), (699, 9), (0, 9)):
        out = torch.full((702,), -7, dtype=torch.int64, device="cuda")
        n = C.c_int64(0)
        assert L.utl_index_stream(C.c_void_p(d.data_ptr()), len(p), C.c_void_p(out.data_ptr()), cap, C.byref(n),
                                  None) == rc
        assert n.value == 700
        assert int((out[cap + 1:] != -7).sum()) == 0
