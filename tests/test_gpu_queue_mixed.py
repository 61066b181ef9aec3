"""Queue launches that mix jobs of the flat kernel with jobs it does not take
(fault jobs that drive a register)."""
import numpy as np
import pytest

from rrtl_gb300 import sim
from rrtl_gb300.workloads import gate_netlist, job_faults, netlist_run_spec

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def netlist(engine):
    d, meta = gate_netlist(n_gates=6000, n_ff=300, n_pi=16, n_po=24, depth=14, seed=12)
    return sim.CompiledDesign(d.to_json(), meta.top), meta


def _job(netlist, lanes, cycles, fused, fault, words=0):
    meta = netlist[1]
    stim, rec = netlist_run_spec(meta, uniform=fault)
    if fused:
        stim = stim + [(meta.regs[0], sim.STIM_RANDOM_UNIFORM, 999)]
    faults = [f for f in job_faults(meta, lanes, 5) if f[1] != meta.regs[0]] if fault else []
    return faults, dict(cycles=cycles, seed=lanes + cycles, stim=stim, record=rec,
                        mode=sim.REC_HASH | sim.REC_TRACE | (sim.REC_DETECT if fault else 0))


def _batch(netlist, lanes, faults, words=0):
    g = sim.GpuBatchSimulator(netlist[0], lanes=lanes)
    g.set_tile_words(words)
    if faults:
        g.set_faults(faults)
    return g


def _submit(ctx, netlist, lanes, cycles, fused=False, fault=False, words=0):
    faults, args = _job(netlist, lanes, cycles, fused, fault, words)
    g = _batch(netlist, lanes, faults, words)
    return g, args, ctx.submit(g, **args)


def test_both_kernels_run_at_the_same_time(netlist):
    """A long job of few tiles on either kernel: a launch of both lasts about as
    long as the longer one (their sum, were one to wait for the other)."""
    ctx = sim.default_context()
    cycles = {False: 4000, True: 4000}
    alone = {}
    for rep in range(2):  # programs are built in the first
        for fused in (False, True):
            job = _submit(ctx, netlist, 64, cycles[fused], fused, fused, words=1)
            ctx.launch()
            ctx.wait()
            alone[fused] = ctx.queue_ms
            if not rep:
                cycles[fused] = max(200, int(cycles[fused] * 20 / alone[fused]))  # 20 ms each
    both = [_submit(ctx, netlist, 64, cycles[fused], fused, fused, words=1) for fused in (False, True)]
    ctx.launch()
    ctx.wait()
    assert all(j.status == sim.JOB_DONE for _, _, j in both + [job])
    assert ctx.queue_ms < 0.75 * sum(alone.values()), (ctx.queue_ms, alone)


@pytest.mark.parametrize("wide", [(False, False), (True, False), (False, True), (True, True)])
def test_mixed_launches_equal_runs_alone(netlist, monkeypatch, wide):
    """Each list short, and longer than the SMs (more blocks than either kernel first gets)."""
    ctx = sim.default_context()
    n = lambda w: 32 * 400 if w else 70
    specs = [(n(wide[0]), 9, False, False, 1), (n(wide[1]), 11, True, True, 1), (300, 40, False, True, 0),
             (33, 60, True, True, 0), (500, 2, False, False, 0), (1000, 30, False, False, 0), (90, 3, False, True, 2)]
    queued = [_submit(ctx, netlist, *s) for s in specs]
    ctx.launch()
    ctx.wait()
    monkeypatch.setenv("RRTL_FLAT", "0")  # alone: on the fused kernel
    for spec, (g, args, job) in zip(specs, queued):
        assert job.status == sim.JOB_DONE
        lanes, cycles, fused, fault, words = spec
        alone = _batch(netlist, lanes, _job(netlist, *spec)[0])
        ref = alone.run(**args)
        for k in ("trace", "hash", "detect"):
            assert (ref[k] is None and job.outputs[k] is None) or np.array_equal(job.outputs[k], ref[k]), (spec, k)
        bits = netlist[1].regs + netlist[1].gate_names[::97]
        assert np.array_equal(g.get_signals_bits(bits), alone.get_signals_bits(bits)), spec
