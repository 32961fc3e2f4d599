"""First use inside a stream capture: any batched call on a device makes every
other batched call there ready to be captured, whatever kernels the two take.
Each pair runs in a process of its own, since the first use of a device happens
once."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = r"""
import sys
sys.path[:0] = [%(root)r, %(tests)r]
import ctypes as C
import numpy as np
import torch
import utlpfor_b200 as U
import oracle_ref as O
from gen import streams
from utlpfor_b200._lib import load

SHAPES = {  # name: (values, kind, uint64, flag)
    "small": (5003, "exc", False, 0),
    "delta": (5003, "sorted", False, 1),
    "large": (128 * 20000 + 5, "exc", False, 0),
    "nopatch": (128 * 20000 + 5, "exc", False, 4),
    "u64": (9001, "for64", True, 0),
}

def inputs(name):
    n, kind, is64, flag = SHAPES[name]
    vals, vo = streams(np.random.default_rng(n), [n], kind, is64=is64)
    want, wbo, _ = O.pack_streams(flag, vals, vo, n_threads=8)
    return vals, vo, flag, want, wbo

def tensors(vals):
    return torch.from_numpy(vals.view(np.int64 if vals.dtype.itemsize == 8 else np.int32)).cuda()

first, then = sys.argv[1:]
L = load()
# everything but the warm-up call's kernels, before it: torch and the stream table
vals, vo, flag, want, wbo = inputs(then)
d = tensors(vals)
codec = U.BatchCodec(vo, flag=flag, is64=vals.dtype.itemsize == 8, tuned=False)
out = torch.empty_like(d)
if first == "unpack":
    v1, vo1, f1, w1, b1 = inputs("small")
    pk, bo = torch.from_numpy(w1).cuda(), torch.from_numpy(b1.view(np.int64)).cuda()
    tvo = torch.from_numpy(vo1.view(np.int64)).cuda()
    tbs = torch.tensor([0, len(b1) - 1], dtype=torch.int64, device="cuda")
    o = torch.empty(len(v1), dtype=torch.int32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    assert L.utl_unpack_batch_u32(p(pk), len(w1), p(bo), p(tvo), p(tbs), 1, len(b1) - 1, p(o), None, None,
                                  C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
else:
    v1, vo1, f1, w1, b1 = inputs(first)
    pb = U.pack_batch(tensors(v1), vo1, f1)
    assert pb.packed[:len(w1)].cpu().numpy().tobytes() == w1.tobytes()
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    codec.pack(d)
    codec.unpack(out)
for _ in range(2):
    codec.packed.zero_()
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert codec.packed[:len(want)].cpu().numpy().tobytes() == want.tobytes()
    assert np.array_equal(codec.block_off.cpu().numpy().view(np.uint64), wbo)
    assert torch.equal(out, d)
assert codec.error_bits() == 0
print("captured")
"""


@pytest.mark.parametrize("first,then", [("small", "large"), ("u64", "large"), ("unpack", "large"), ("large", "small"),
                                        ("unpack", "delta"), ("unpack", "u64"), ("large", "u64"),
                                        ("unpack", "nopatch")])
def test_capture_after_another_route(first, then):
    code = CHILD % {"root": os.path.dirname(HERE), "tests": HERE}
    out = subprocess.run([sys.executable, "-c", code, first, then], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, (out.stdout + out.stderr)[-3000:]
    assert "captured" in out.stdout
