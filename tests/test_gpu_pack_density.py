"""Large NoPatch batches take the launches that suit their block size: two for
blocks of which a tile does not fit the one-launch pack's image, one for others,
by the mean block of the batch before.  In a process of its own: the first batch
of a device has none before it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = r"""
import sys
sys.path[:0] = [%(root)r, %(tests)r]
import numpy as np
import torch
import utlpfor_b200 as U
import oracle_ref as O
from utlpfor_b200._lib import load

L = load()
assert L.utl_get_knob(2) == 3
rng = np.random.default_rng(1)
N = 128 * 16384 + 77

def batch(bits, flag):
    v = rng.integers(0, 2**bits, N, dtype=np.uint64).astype(np.uint32)
    vo = np.array([0, 700003, N], np.uint64)
    want, wbo, _ = O.pack_streams(flag, v, vo, n_threads=8)
    d = torch.from_numpy(v.view(np.int32)).cuda()
    codec = U.BatchCodec(vo, flag=flag, tuned=False)
    def go():
        codec.packed.zero_()
        n0 = L.utl_launch_count()
        codec.pack(d)
        n = L.utl_launch_count() - n0
        torch.cuda.synchronize()
        assert codec.error_bits() == 0
        assert codec.packed[:len(want)].cpu().numpy().tobytes() == want.tobytes()
        assert np.array_equal(codec.block_off.cpu().numpy().view(np.uint64), wbo)
        return n
    return go

narrow, wide, patched, deltas = batch(8, 4), batch(32, 4), batch(32, 0), batch(12, 5)
assert narrow() == 1             # nothing known yet
assert narrow() == 1             # 132 bytes a block
assert wide() == 1               # goes by the narrow one
assert wide() == 2               # 516 bytes a block
assert patched() == 1            # never asked; leaves what NoPatch goes by alone
assert wide() == 2
assert narrow() == 2
assert narrow() == 1
assert deltas() == 1            # goes by the narrow one
assert deltas() == 2            # signed 13-bit differences: 260 bytes a block
print("routes ok")
"""


def test_route_follows_block_size():
    code = CHILD % {"root": os.path.dirname(HERE), "tests": HERE}
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, (out.stdout + out.stderr)[-3000:]
    assert "routes ok" in out.stdout
