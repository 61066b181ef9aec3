"""The flat gate kernel at every shape against the bit-parallel oracle: ragged
lane counts around its tiles, every record form, more stimulus and record
words than its service threads hold in registers, registers left on the
commit list, a recorded input, and runs split in two."""
import numpy as np
import pytest

from oracle import binding as ob
from rrtl_gb300 import sim
from rrtl_gb300.workloads import gate_netlist, netlist_run_spec

from .helpers import oracle_bp_run

pytestmark = pytest.mark.gpu

SHAPES = {"111": 1, "211": 2, "411": 4, "421": 8, "431": 12, "422": 16}


@pytest.fixture(scope="module")
def wide(engine):
    """200 inputs and outputs: at 16 words a tile has 3,200 stimulus and record words."""
    d, meta = gate_netlist(n_gates=4000, n_ff=300, n_pi=200, n_po=200, depth=9, seed=8)
    js = d.to_json()
    return sim.CompiledDesign(js, meta.top), meta, ob.OracleDesign(js, meta.top)


def _ref(od, lanes, cycles, seed, stim, rec, mode, **kw):
    return oracle_bp_run(od, lanes, cycles, seed, [(od.signal(n), k, p) for n, k, p in stim],
                         [od.signal(r) for r in rec], mode, **kw)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("lanes", [1, 500, 32 * 16 * 3 + 7])
def test_shapes_equal_the_oracle(wide, monkeypatch, shape, lanes):
    cd, meta, od = wide
    monkeypatch.setenv("RRTL_FLAT", shape)
    stim, rec = netlist_run_spec(meta)
    mode = sim.REC_TRACE | sim.REC_HASH | sim.REC_DETECT
    g = sim.GpuBatchSimulator(cd, lanes=lanes)
    res = g.run(13, seed=5, stim=stim, record=rec, mode=mode, lane_base=64)
    assert g.tile_words == {12: 4, 16: 8}.get(SHAPES[shape], SHAPES[shape])
    ref = _ref(od, lanes, 13, 5, stim, rec, mode, lane_base=64)
    for k in ("trace", "hash", "detect"):
        assert np.array_equal(res[k], ref[k]), k
    ref["sim"].settle()
    for n in meta.regs[::17] + meta.gate_names[::101] + meta.outputs[::9]:
        assert np.array_equal(g.get_signal_bits(n), ref["sim"].get_bits(od.signal(n))), n


@pytest.mark.parametrize("shape", ["111", "421", "422"])
def test_trace_input_and_recorded_input(wide, monkeypatch, shape):
    """Stimulus from a trace; a recorded net that is itself stimulated."""
    cd, meta, od = wide
    monkeypatch.setenv("RRTL_FLAT", shape)
    lanes, cycles = 300, 11
    words = (lanes + 31) // 32
    tr = np.random.default_rng(4).integers(0, 1 << 32, (cycles, len(meta.inputs), words), dtype=np.uint32)
    stim = [(meta.rst, sim.STIM_PULSE, 1)] + [(p, sim.STIM_TRACE, i) for i, p in enumerate(meta.inputs)]
    rec = meta.outputs[:40] + meta.inputs[:5]
    g = sim.GpuBatchSimulator(cd, lanes=lanes)
    res = g.run(cycles, seed=1, stim=stim, record=rec, mode=sim.REC_TRACE | sim.REC_HASH, input_trace=tr)
    assert g.tile_words == {12: 4, 16: 8}.get(SHAPES[shape], SHAPES[shape])
    ref = _ref(od, lanes, cycles, 1, stim, rec, 3, input_trace=tr)
    assert np.array_equal(res["trace"], ref["trace"]) and np.array_equal(res["hash"], ref["hash"])


@pytest.mark.parametrize("shape", ["211", "422"])
def test_runs_continue_from_the_state_they_leave(wide, monkeypatch, shape):
    cd, meta, od = wide
    monkeypatch.setenv("RRTL_FLAT", shape)
    stim, rec = netlist_run_spec(meta)
    hold = [(meta.rst, sim.STIM_CONST, 0)]  # inputs keep the values the first run left
    g = sim.GpuBatchSimulator(cd, lanes=700)
    a = g.run(6, seed=2, stim=stim, record=rec, mode=sim.REC_HASH)["hash"]
    b = g.run(7, seed=2, stim=hold, record=rec, mode=sim.REC_HASH)["hash"]
    monkeypatch.setenv("RRTL_FLAT", "0")
    f = sim.GpuBatchSimulator(cd, lanes=700)
    assert np.array_equal(a, f.run(6, seed=2, stim=stim, record=rec, mode=sim.REC_HASH)["hash"])
    assert np.array_equal(b, f.run(7, seed=2, stim=hold, record=rec, mode=sim.REC_HASH)["hash"])
    for n in meta.regs[::29] + meta.inputs[::31] + meta.gate_names[::211]:
        assert np.array_equal(g.get_signal_bits(n), f.get_signal_bits(n)), n


@pytest.mark.parametrize("shape", ["111", "411", "422"])
def test_registers_on_the_commit_list(engine, monkeypatch, shape):
    """A shift chain is longer than the levels, so part of it commits after them."""
    from rrtl_gb300.builder import Design, mux, uint

    d = Design()
    m = d.module("Chain")
    clk, rst, en, x = (m.input(n, uint(1)) for n in ("clk", "rst", "en", "x"))
    regs = [m.reg(f"r{k}", uint(1)) for k in range(260)]
    for k, r in enumerate(regs):
        m.clock(r, clk)
        if k % 3:
            m.reset(r, rst, k % 2)
        m.next(r, mux(en, regs[k - 1] if k else x, r))
    for k in range(4):
        o = m.output(f"o{k}", uint(1))
        m.assign(o, regs[50 * k + 9] ^ regs[259])
    js = d.to_json()
    cd, od = sim.CompiledDesign(js, "Chain"), ob.OracleDesign(js, "Chain")
    monkeypatch.setenv("RRTL_FLAT", shape)
    monkeypatch.setenv("RRTL_GATE_JIT", "0")
    stim = [("clk", sim.STIM_CONST, 1), ("rst", sim.STIM_PULSE, 2), ("en", sim.STIM_RANDOM, 1), ("x", sim.STIM_RANDOM, 2)]
    rec = [f"o{k}" for k in range(4)]
    g = sim.GpuBatchSimulator(cd, lanes=1000)
    res = g.run(60, seed=9, stim=stim, record=rec, mode=3)
    assert g.tile_words != 0
    ref = _ref(od, 1000, 60, 9, stim, rec, 3)
    assert np.array_equal(res["trace"], ref["trace"]) and np.array_equal(res["hash"], ref["hash"])


@pytest.mark.parametrize("shape", SHAPES)
def test_stuck_at_faults(wide, monkeypatch, shape):
    """Many faults on few lanes (more than a 32-force window per warp), on
    wires, registers, outputs, several on one lane, two on one net."""
    from rrtl_gb300.workloads import Rng

    cd, meta, od = wide
    monkeypatch.setenv("RRTL_FLAT", shape)
    rng = Rng(int(shape))
    lanes, cycles = 540, 14
    sites = meta.gate_names + meta.regs + meta.outputs
    faults = [(l, sites[rng.below(len(sites))], rng.below(2)) for l in range(lanes) if l % 32 for _ in range(1 + 8 * (l < 64))]
    faults += [(33, meta.regs[3], 1), (33, meta.regs[3], 0), (34, meta.gate_names[5], 0), (34, meta.gate_names[5], 1)]
    stim, rec = netlist_run_spec(meta, uniform=True)
    mode = sim.REC_TRACE | sim.REC_HASH | sim.REC_DETECT
    g = sim.GpuBatchSimulator(cd, lanes=lanes)
    g.set_faults(faults)
    res = g.run(cycles, seed=3, stim=stim, record=rec, mode=mode)
    assert g.tile_words == {12: 4, 16: 8}.get(SHAPES[shape], SHAPES[shape])
    ref = _ref(od, lanes, cycles, 3, stim, rec, mode, faults=[(l, od.signal(s), v) for l, s, v in faults])
    for k in ("trace", "hash", "detect"):
        assert np.array_equal(res[k], ref[k]), k
    for n in meta.regs:
        assert np.array_equal(g.get_signal_bits(n), ref["sim"].get_bits(od.signal(n))), n


def test_queue_of_flat_and_fused_jobs(wide, monkeypatch):
    """One launch of jobs of every size (a long one on one lane, wide ones,
    one too short for the flat kernel, fault jobs, an explicit tile width)
    equals the same runs alone on the fused kernel."""
    from rrtl_gb300.workloads import job_faults

    cd, meta, od = wide
    jobs = [(1, 400, 0, 0), (3000, 20, 0, 0), (77, 2, 0, 0), (640, 30, 1, 0), (2048, 9, 1, 0), (33, 50, 0, 2), (900, 8, 0, 8)]
    out = {}
    for flat in ("", "0"):
        monkeypatch.setenv("RRTL_FLAT", flat)
        ctx = sim.default_context()
        queued, keep = [], []
        for i, (lanes, cycles, fault, words) in enumerate(jobs):
            g = sim.GpuBatchSimulator(cd, lanes=lanes)
            g.set_tile_words(words)
            if fault:
                g.set_faults(job_faults(meta, lanes, i))
            stim, rec = netlist_run_spec(meta, uniform=bool(fault))
            mode = sim.REC_HASH | sim.REC_TRACE | (sim.REC_DETECT if fault else 0)
            keep.append(g)
            if flat == "":
                queued.append(ctx.submit(g, cycles, seed=i, stim=stim, record=rec, mode=mode))
            else:
                queued.append(g.run(cycles, seed=i, stim=stim, record=rec, mode=mode))
        if flat == "":
            ctx.launch()
            ctx.wait()
            assert [j.status for j in queued] == [sim.JOB_DONE] * len(jobs)
            queued = [j.outputs for j in queued]
        out[flat] = [(r, g.get_signals_bits(meta.regs + meta.gate_names[::97])) for r, g in zip(queued, keep)]
    for (a, sa), (b, sb) in zip(out[""], out["0"]):
        for k in ("trace", "hash", "detect"):
            assert (a[k] is None and b[k] is None) or np.array_equal(a[k], b[k]), k
        assert np.array_equal(sa, sb)


@pytest.mark.parametrize("lanes", [33, 32 * 16 * 3 + 7, 32 * 2500])
def test_closing_settle_writes_every_signal(wide, monkeypatch, lanes):
    """Lanes for its widths of 1, 4 and 8 words: each signal as the fused kernel leaves it."""
    cd, meta, od = wide
    stim, rec = netlist_run_spec(meta)
    got = []
    for flat in ("411", "0"):
        monkeypatch.setenv("RRTL_FLAT", flat)
        g = sim.GpuBatchSimulator(cd, lanes=lanes)
        g.run(5, seed=4, stim=stim, record=rec, mode=sim.REC_HASH)
        step = 1 if lanes < 5000 else 41
        got.append([g.get_signal_bits(n) for n in (meta.inputs + meta.regs + meta.gate_names)[::step]])
    assert all(np.array_equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("shape,words", [("111", 153), ("111", 301), ("211", 500), ("422", 16 * 171)])
@pytest.mark.parametrize("cycles", [4, 11])
def test_tiles_split_between_blocks(wide, monkeypatch, shape, words, cycles):
    """More tiles than SMs and no multiple: blocks share tiles, every record form, faults detected in either part."""
    cd, meta, od = wide
    monkeypatch.setenv("RRTL_FLAT", shape)
    stim, rec = netlist_run_spec(meta)
    lanes = 32 * words - 9
    g = sim.GpuBatchSimulator(cd, lanes=lanes)
    res = g.run(cycles, seed=6, stim=stim, record=rec[:40], mode=sim.REC_TRACE | sim.REC_HASH)
    ref = _ref(od, lanes, cycles, 6, stim, rec[:40], 3)
    assert np.array_equal(res["hash"], ref["hash"]) and np.array_equal(res["trace"], ref["trace"])
    uni = [(n, sim.STIM_RANDOM_UNIFORM if k == sim.STIM_RANDOM else k, p) for n, k, p in stim]
    got = []
    for flat in (shape, "0"):
        monkeypatch.setenv("RRTL_FLAT", flat)
        f = sim.GpuBatchSimulator(cd, lanes=lanes)
        f.set_faults([(ln, meta.gate_names[ln % len(meta.gate_names)], ln & 1) for ln in range(1, lanes, 7) if ln % 32])
        got.append(f.run(cycles, seed=6, stim=uni, record=rec, mode=sim.REC_DETECT)["detect"])
    assert np.array_equal(*got) and (got[0] != 0xFFFFFFFF).any()


@pytest.mark.parametrize("shape", ["111", "211"])
def test_more_rows_than_byte_offsets_name(engine, monkeypatch, shape):
    """Over 16,384 one-word rows: entries hold row numbers instead of byte offsets."""
    d, meta = gate_netlist(n_gates=20_000, n_ff=16_500, n_pi=8, n_po=8, depth=6, seed=3)
    js = d.to_json()
    od = ob.OracleDesign(js, meta.top)
    monkeypatch.setenv("RRTL_FLAT", shape)
    stim, rec = netlist_run_spec(meta)
    g = sim.GpuBatchSimulator(sim.CompiledDesign(js, meta.top), lanes=70)
    res = g.run(6, seed=9, stim=stim, record=rec, mode=sim.REC_HASH)
    assert g.tile_words == int(shape[0])
    assert np.array_equal(res["hash"], _ref(od, 70, 6, 9, stim, rec, 2)["hash"])


@pytest.mark.parametrize("name", ["401", "128", "412", "999", "abc"])
def test_unknown_shapes_are_refused(wide, monkeypatch, name):
    """A forced shape that is not built is an error of the run, not an index into the shapes' tables."""
    cd, meta, od = wide
    monkeypatch.setenv("RRTL_FLAT", name)
    stim, rec = netlist_run_spec(meta)
    g = sim.GpuBatchSimulator(cd, lanes=40)
    with pytest.raises(sim.RrtlError) as e:
        g.run(5, seed=1, stim=stim, record=rec, mode=sim.REC_HASH)
    assert e.value.code == "E_GPU_FLAT"
    monkeypatch.delenv("RRTL_FLAT")
    res = g.run(5, seed=1, stim=stim, record=rec, mode=sim.REC_HASH)
    assert np.array_equal(res["hash"], _ref(od, 40, 5, 1, stim, rec, 2)["hash"])
