"""The stream indexer's answer for a stream with a bad block: the status and the
index of the first one, as the oracle's walk gives them, from the two launches
that index a good stream; around the edges of regions (32256 bytes) and teams
(1008), with more bad blocks behind the first, and for streams of noise."""
import ctypes as C

import numpy as np
import pytest

import oracle_ref as O
from gen import streams

pytestmark = pytest.mark.gpu

REGION, TEAM = 32256, 1008


def _index(torch, L, buf, skew, p, cap):
    d = buf[skew:skew + len(p)]
    d.copy_(torch.from_numpy(p))
    out = torch.empty(cap + 1, dtype=torch.int64, device="cuda")
    n = C.c_int64(-1)
    n0 = L.utl_launch_count()
    rc = L.utl_index_stream(C.c_void_p(d.data_ptr()), len(p), C.c_void_p(out.data_ptr()), cap, C.byref(n), None)
    return rc, n.value, L.utl_launch_count() - n0, out


def _damage(p, o, how):
    if how == "reserved":
        p[o + 2] |= 0x14
    elif how == "count":
        p[o] = 200
    else:
        p[o + 1] |= 0x1F


@pytest.mark.parametrize("how", ["reserved", "count", "width"])
@pytest.mark.parametrize("skew", [0, 7])
@pytest.mark.parametrize("kind,flag,is64", [("exc", 0, False), ("sorted", 1, False), ("zero", 0, False),
                                            ("full", 4, False), ("full", 0, True), ("walk", 1, True)])
def test_first_bad_block(kind, flag, is64, skew, how):
    import torch

    from utlpfor_b200._lib import load
    L = load()
    n = 128 * (20000 if kind == "zero" else 330)
    vals, vo = streams(np.random.default_rng(n + flag), [n], kind, is64=is64)
    packed, bo, _ = O.pack_streams(flag, vals, vo)
    bo = bo.astype(np.int64)
    nb = len(bo) - 1
    buf = torch.zeros(len(packed) + 64, dtype=torch.uint8, device="cuda")
    at = {0, 1, nb // 2, nb - 2, nb - 1}
    for edge in (TEAM, REGION - TEAM, REGION, REGION + TEAM, 2 * REGION):
        i = int(np.searchsorted(bo, edge))
        at.update(b for b in (i - 1, i, i + 1) if 0 <= b < nb)
    rng = np.random.default_rng(5)
    for b in sorted(at):
        p = packed.copy()
        _damage(p, int(bo[b]), how)
        for later in rng.integers(b, nb, 3):
            _damage(p, int(bo[later]), how)
        _, err, want = O.index_stream(p)
        assert err != O.OK and want == b
        rc, got, launches, _ = _index(torch, L, buf, skew, p, nb)
        assert (rc, got) == (err, want)
        assert launches == 2
    # cut inside the last block
    for cut in (1, min(3, int(bo[nb] - bo[nb - 1]) - 1)):
        p = packed[:-cut]
        _, err, want = O.index_stream(p)
        rc, got, launches, _ = _index(torch, L, buf, skew, p, nb)
        assert (rc, got, launches) == (err, want, 2)
    # and the good stream behind them
    rc, got, _, out = _index(torch, L, buf, skew, packed, nb)
    assert (rc, got) == (0, nb) and np.array_equal(out.cpu().numpy(), bo)


@pytest.mark.parametrize("seed", range(6))
def test_noise(seed):
    import torch

    from utlpfor_b200._lib import load
    L = load()
    rng = np.random.default_rng(seed)
    n = int(rng.integers(1, 5 * REGION))
    p = rng.integers(0, 256, n, dtype=np.uint8)
    if seed % 2:  # a good start, noise from somewhere on
        vals, vo = streams(rng, [60000], "exc")
        good, _, _ = O.pack_streams(0, vals, vo)
        p = np.concatenate([good[:int(rng.integers(1, len(good)))], p])
    want_off, err, want = O.index_stream(p)
    buf = torch.zeros(len(p) + 64, dtype=torch.uint8, device="cuda")
    rc, got, _, out = _index(torch, L, buf, seed % 16, p, len(p) // 4 + 1)
    if err == O.OK:
        assert (rc, got) == (0, len(want_off) - 1) and list(out[:got + 1].cpu().numpy()) == list(want_off)
    else:
        assert (rc, got) == (err, want)
