"""The exception writer of the two-launch pack (utl_qpack.cuh), compiled with
the host compiler and run a thread per lane under the thread sanitizer
(tests/pack_exceptions_check.cc): right bytes, and no byte shared by two lanes
without a barrier between them.  No GPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "utlpfor_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_lanes_share_no_bytes(tmp_path):
    with open(os.path.join(CSRC, "utl_qpack.cuh")) as f:
        text = "".join(ln for ln in f if not ln.startswith(("#include", "#pragma once")))
    (tmp_path / "qpack_host.h").write_text(text)
    exe = str(tmp_path / "check")
    built = subprocess.run(["g++", "-O1", "-g", "-std=c++20", "-pthread", "-fsanitize=thread", "-Wno-unknown-pragmas",
                            "-I", str(tmp_path), os.path.join(HERE, "pack_exceptions_check.cc"), "-o", exe],
                           capture_output=True, text=True)
    if built.returncode and "tsan" in built.stderr:
        pytest.skip("no thread sanitizer")
    assert built.returncode == 0, built.stderr
    # a fixed address layout where that can be had: some kernels randomise more than the sanitizer can map
    fixed = ["setarch", "-R"] if shutil.which("setarch") and subprocess.run(["setarch", "-R", "true"]).returncode == 0 else []
    run = fixed + [exe]
    out = subprocess.run(run, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, (out.stdout + out.stderr)[-3000:]
    assert out.stdout.startswith("ok "), out.stdout
