"""The autotuner's choice: kept when a measurement fails, made on the kernel that longer runs take."""
import numpy as np
import pytest

from oracle import binding as ob
from rrtl_gb300 import sim
from rrtl_gb300.workloads import gate_netlist, netlist_run_spec

from .helpers import oracle_bp_run

pytestmark = pytest.mark.gpu

LANES = 4096


@pytest.fixture()
def design(engine):
    d, meta = gate_netlist(n_gates=9000, n_ff=300, n_pi=16, n_po=16, depth=12, seed=6)
    js = d.to_json()
    return sim.CompiledDesign(js, meta.top), meta, ob.OracleDesign(js, meta.top)


def _width(design, lanes=LANES, cycles=6):
    """Tile width of a run, whose hashes are the oracle's."""
    cd, meta, od = design
    stim, rec = netlist_run_spec(meta)
    g = sim.GpuBatchSimulator(cd, lanes=lanes)
    res = g.run(cycles, seed=3, stim=stim, record=rec, mode=sim.REC_HASH)
    ref = oracle_bp_run(od, lanes, cycles, 3, [(od.signal(n), k, p) for n, k, p in stim], [od.signal(r) for r in rec], 2)
    assert np.array_equal(res["hash"], ref["hash"])
    return g.tile_words


@pytest.mark.parametrize("words", [0, 1, 2])
def test_a_failed_autotune_keeps_the_choice(design, monkeypatch, words):
    """words 0: untuned before."""
    cd = design[0]
    if words:
        table = [{"case": "c", "lanes": LANES, "steps": 8, "tile_words": words, "autotune_metric": "kernel_ms",
                  "autotune_metric_ns": 1}]
        assert cd.autotune_apply(table, "c", LANES, 8) == words
    before = _width(design)
    assert not words or before == words
    monkeypatch.setenv("RRTL_FLAT", "999")  # no such shape: every candidate's run is an error
    with pytest.raises(sim.RrtlError) as e:
        cd.autotune(LANES, cycles=8)
    assert e.value.code == "E_GPU_FLAT"
    monkeypatch.delenv("RRTL_FLAT")
    assert _width(design) == before


def test_few_cycles_are_measured_on_the_flat_kernel(design, monkeypatch):
    cd = design[0]
    monkeypatch.setenv("RRTL_FLAT", "999")
    with pytest.raises(sim.RrtlError):
        cd.autotune(LANES, cycles=2)
    monkeypatch.delenv("RRTL_FLAT")
    best, ms = cd.autotune(LANES, cycles=2)
    assert best in (0, 1, 2, 4, 8) and ms > 0
    assert _width(design, cycles=6) == best
    assert _width(design, cycles=2) == best
