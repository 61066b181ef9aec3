"""The gate kernels' detection state at the start of a run: read from one
entry a lane, never past the lanes a caller's buffer has (tests/native/detected_lanes.cpp)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def prog(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("native") / "detected_lanes")
    subprocess.run(["g++", "-O0", "-std=c++17", "-o", exe, os.path.join(HERE, "native", "detected_lanes.cpp")], check=True)
    return exe


@pytest.mark.parametrize("lanes", [1, 31, 32, 33, 540, 1023, 1024, 1025])
@pytest.mark.parametrize("step", [1, 3])
def test_reads_end_with_the_lanes(prog, lanes, step):
    r = subprocess.run([prog, str(lanes), str(step)], capture_output=True, text=True)
    assert r.returncode == 0
    got = [int(x) for x in r.stdout.split()]
    words = (lanes + 31) // 32
    want = [sum(1 << b for b in range(32) if w * 32 + b < lanes and (w * 32 + b) % step == 0) for w in range(words)]
    assert got == want + [0, 0, 0]


def test_no_kernel_reads_the_buffer_by_itself():
    """Every kernel takes its starting state from detected_lanes (the plain one reads a lane that it found to differ)."""
    csrc = os.path.join(os.path.dirname(HERE), "rrtl_gb300", "csrc")
    for f in ("gate_flat.h", "gate_fused.h", "gate_jit.cpp"):
        text = open(os.path.join(csrc, f)).read()
        assert "detected_lanes(R.detect," in text and "] != 0xFFFFFFFFu) det" not in text, f
