"""Designs that prefer the compiled gate kernel, in runs that it does not take:
the flat kernel runs them. A forced one-word tile tells it from the fused
kernel, which picks wide tiles at these lane counts."""
import numpy as np
import pytest

from oracle import binding as ob
from rrtl_gb300 import sim
from rrtl_gb300.workloads import gate_netlist, narrow_alu, netlist_run_spec

from .helpers import oracle_bp_run

pytestmark = pytest.mark.gpu

LANES, CYCLES = 32 * 1200 + 5, 9


def _check(js, top, stim, rec, width, cycles=CYCLES):
    cd, od = sim.CompiledDesign(js, top), ob.OracleDesign(js, top)
    g = sim.GpuBatchSimulator(cd, lanes=LANES)
    res = g.run(cycles, seed=8, stim=stim, record=rec, mode=sim.REC_HASH | sim.REC_TRACE)
    assert g.tile_words == width
    ref = oracle_bp_run(od, LANES, cycles, 8, [(od.signal(n), k, p) for n, k, p in stim], [od.signal(r) for r in rec], 3)
    assert np.array_equal(res["hash"], ref["hash"]) and np.array_equal(res["trace"], ref["trace"])


def _netlist(n_po):
    d, meta = gate_netlist(n_gates=170, n_ff=20, n_pi=9, n_po=n_po, depth=6, seed=12)
    return (d.to_json(), meta.top) + netlist_run_spec(meta)


@pytest.mark.parametrize("n_po,width", [(64, 0), (65, 1)])
def test_more_records_than_the_compiled_kernel_takes(engine, monkeypatch, n_po, width):
    monkeypatch.setenv("RRTL_FLAT", "111")
    _check(*_netlist(n_po), width)


def test_more_inputs_than_the_compiled_kernel_takes(engine, monkeypatch):
    """The bit planes of a 62-bit datapath: 66 inputs, two cells a level."""
    monkeypatch.setenv("RRTL_FLAT", "111")
    w = 62
    js = sim.bitslice_json(narrow_alu(w), "Alu")
    stim = [("clk[0]", sim.STIM_CONST, 1), ("rst[0]", sim.STIM_PULSE, 1)]
    stim += [(f"din[{p}]", sim.STIM_RANDOM, p) for p in range(w)] + [(f"sel[{p}]", sim.STIM_RANDOM, 100 + p) for p in range(2)]
    _check(js, "Alu", stim, [f"out[{p}]" for p in range(16)] + ["flag[0]"], 1, cycles=6)


def test_compiled_kernel_switched_off(engine, monkeypatch):
    monkeypatch.setenv("RRTL_GATE_JIT", "0")
    monkeypatch.setenv("RRTL_FLAT", "111")
    _check(*_netlist(20), 1)
    _check(*_netlist(20), 8, cycles=3)  # too short for the flat kernel


def test_an_invalid_run_is_refused_before_anything_is_built(engine):
    js, top, stim, rec = _netlist(20)
    g = sim.GpuBatchSimulator(js, top, 64)
    for kw in (dict(mode=sim.REC_HASH, record=[]), dict(stim=[(rec[0], sim.STIM_CONST, 1)]),
               dict(stim=[(stim[0][0], 9, 1)]), dict(stim=[(stim[0][0], sim.STIM_TRACE, 0)]), dict(lane_base=5)):
        with pytest.raises(sim.RrtlError):
            g.run(5, **{"stim": stim, "record": rec, **kw})
