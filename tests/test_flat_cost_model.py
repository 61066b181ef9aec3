"""The cost model that chooses tile shapes of the flat kernel against clocks
measured on the device (one wave of tiles, 2,070 MHz): netlists of one family
with levels and gates varied apart, so that no term stands in for another."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from rrtl_gb300.workloads import gate_netlist

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "rrtl_gb300", "csrc")
# V, N, Q, narrow: one and two words in the queue and in runs, then the wide tiles
SHAPES = [(1, 1, 1, 0), (1, 1, 1, 1), (2, 1, 1, 0), (2, 1, 1, 1), (4, 1, 1, 0), (4, 2, 1, 0), (4, 3, 1, 0), (4, 2, 2, 0)]
MEASURED = {  # (gates, depth): clocks a tile-cycle per shape (None: the tile does not fit)
    (3000, 40): (10296, 10691, 11408, 10917, 13663, 17554, 24153, 24573),
    (10000, 10): (7388, 7358, 8857, 9132, 10914, 16062, 21186, 21988),
    (10000, 40): (11820, 12051, 13746, 13715, 17513, 25217, 32456, 36908),
    (10000, 160): (34073, 34769, 36712, 36911, 44455, 56818, 77098, 77895),
    (20000, 40): (14720, 14978, 17344, 17534, 22756, 33734, 43997, 52441),
    (50000, 10): (17222, 16188, 20829, 19969, 26995, None, None, None),
    (50000, 40): (24878, 23407, 29255, 27926, 36575, 56207, 76508, 95796),
    (50000, 160): (43866, 44458, 49251, 49245, 62723, 93773, 123000, 135615),
}


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("native") / "libflat_cost.so")
    src = [os.path.join(HERE, "native", "flat_cost.cpp")] + [
        os.path.join(CSRC, f) for f in ("flatprog.cpp", "gateprog.cpp", "design.cpp", "lower.cpp")]
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", lib] + src, check=True)
    L = ctypes.CDLL(lib)
    P = ctypes.POINTER
    L.flat_costs.argtypes = [ctypes.c_char_p, ctypes.c_size_t, ctypes.c_char_p, ctypes.c_uint32, P(ctypes.c_uint32),
                             P(ctypes.c_double)]
    return L


@pytest.mark.parametrize("gates,depth", MEASURED)
def test_within_an_eighth_of_the_measured_clocks(model, gates, depth):
    """(The fit itself is within 8% of the one- and two-word tiles and 11% of the others.)"""
    d, meta = gate_netlist(n_gates=gates, n_ff=max(64, gates * 2048 // 50_000), depth=depth, seed=2)
    js = d.to_json().encode()
    sh, out = np.array(SHAPES, dtype=np.uint32).ravel(), np.zeros(len(SHAPES))
    assert model.flat_costs(js, len(js), meta.top.encode(), len(SHAPES),
                            sh.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)),
                            out.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0
    off = {s: round(c / m - 1, 3) for s, c, m in zip(SHAPES, out, MEASURED[(gates, depth)]) if m}
    assert max(map(abs, off.values())) <= 0.125, off
