"""Performance cases: the runs a user of this framework makes, through its public entry points.

Every case is one call sequence of the Python API over the C ABI, with host
buffers in and out, as a test bench, a fault-simulation job or a job stream
makes it. A program compiles a design once and then makes many batches of it,
so compiled designs are kept in `_DESIGNS`; a batch (lane state, stimulus
seed, memories, faults) is made anew by every prepare().

Outputs are whole numbers (hashes, traces, detection cycles, register bits):
two correct implementations agree on every bit, so `exact` has no 64-bit
floating values to give and returns None.
"""
from __future__ import annotations

import json
import math
import os

import numpy as np

from rrtl_gb300 import sim
from rrtl_gb300.workloads import (cpu_rom_hashed, counter, gate_netlist, job_faults, log_uniform_int, narrow_alu,
                                  netlist_run_spec, pipelined_cpu, replicated_datapath, Rng)

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_DESIGNS = {}


def listed():
    return [
        # a test bench that drives the README counter clock by clock: inputs in, tick, output back
        {"name": "counter_tick", "kind": "tick", "lanes": 4},
        # the counter's whole output trace brought to the host (1,024 lanes x 10,000 cycles of the benchmark)
        {"name": "counter_trace", "kind": "counter", "lanes": 1024, "cycles": 10_000},
        # the 8-stage pipelined CPU with a program per lane (a quarter of the benchmark's 20,000 cycles)
        {"name": "cpu8", "kind": "cpu", "lanes": 16_384, "cycles": 5_000},
        # the small netlist of the reference's own GPU benchmark at its lane count, hashed per cycle
        {"name": "crc32", "kind": "crc32", "lanes": 262_144, "cycles": 1_000},
        # the headline workload: 50,000 gates, 65,536 lanes, final flip-flops read back
        {"name": "netlist_full", "kind": "netlist", "gates": 50_000, "lanes": 65_536, "cycles": 1_000, "io": "state"},
        # the same netlist debugged on a handful of lanes with a full output trace: latency of a small batch
        {"name": "netlist_few", "kind": "netlist", "gates": 50_000, "lanes": 200, "cycles": 100, "io": "trace"},
        # a caller with its own stimulus: input trace in, output trace out, ragged lane count
        {"name": "netlist_replay", "kind": "netlist", "gates": 50_000, "lanes": 5_003, "cycles": 200, "io": "replay"},
        # a large netlist (narrow tiles), ragged lane count
        {"name": "netlist_200k", "kind": "netlist", "gates": 200_000, "lanes": 10_007, "cycles": 100, "io": "state"},
        # fault simulation: a stuck-at fault on all but one lane of every 32, first detecting cycle per lane
        {"name": "faults", "kind": "fault", "gates": 20_000, "lanes": 16_384, "cycles": 300},
        # an uneven stream of jobs (sizes, lanes, cycles, some of them fault jobs) in one queue launch
        {"name": "job_queue", "kind": "queue", "jobs": 24, "gates_hi": 60_000, "lanes_hi": 8_192, "cycles_hi": 600},
        # a multi-bit datapath run as bit planes
        {"name": "bitslice_alu", "kind": "bitslice", "width": 16, "lanes": 65_536, "cycles": 500},
        # 64 instances of one datapath folded into the lane axis, host input trace, outputs traced
        {"name": "folded_datapath", "kind": "fold", "instances": 64, "lanes": 256, "cycles": 200},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["netlist"] * 5 + ["fault", "fault", "queue", "crc32", "cpu", "counter", "tick", "bitslice", "fold"])
    if kind == "netlist":
        gates, lanes = _log(rng, 2_000, 200_000), _log(rng, 32, 65_536)
        top = max(20, min(1_000, int(4e11 / (gates * lanes))))
        io = rng.choice(["state", "trace", "replay"])
        if io != "state":  # 128 or 64 recorded columns of a host trace: at most some 64 MB
            top = max(20, min(top, int(1e9 / (8 * lanes))))
        return {"kind": kind, "gates": gates, "lanes": lanes, "cycles": _log(rng, 20, top), "io": io}
    if kind == "fault":
        gates, lanes = _log(rng, 2_000, 60_000), _log(rng, 64, 32_768)
        return {"kind": kind, "gates": gates, "lanes": lanes,
                "cycles": _log(rng, 20, max(21, min(600, int(1e11 / (gates * lanes)))))}
    if kind == "queue":
        return {"kind": kind, "jobs": rng.randint(4, 30), "gates_hi": _log(rng, 10_000, 80_000),
                "lanes_hi": _log(rng, 256, 8_192), "cycles_hi": _log(rng, 100, 600)}
    if kind == "crc32":
        return {"kind": kind, "lanes": _log(rng, 32, 1_000_000), "cycles": _log(rng, 50, 1_000)}
    if kind == "cpu":
        return {"kind": kind, "lanes": _log(rng, 32, 32_768), "cycles": _log(rng, 100, 5_000)}
    if kind == "counter":
        return {"kind": kind, "lanes": _log(rng, 32, 4_096), "cycles": _log(rng, 100, 4_000)}
    if kind == "tick":
        return {"kind": kind, "lanes": _log(rng, 1, 16_384)}
    if kind == "bitslice":
        return {"kind": kind, "width": rng.randint(4, 24), "lanes": _log(rng, 64, 262_144),
                "cycles": _log(rng, 50, 500)}
    return {"kind": "fold", "instances": rng.choice([4, 7, 16, 33, 64]), "lanes": _log(rng, 16, 512),
            "cycles": _log(rng, 20, 200)}


# ------------------------------------------------------------------ designs --
def _design(key, build):
    if key not in _DESIGNS:
        _DESIGNS[key] = build()
    return _DESIGNS[key]


def _netlist(gates):
    """The 50,000-gate family: flip-flops in proportion, 64 inputs and outputs, depth 40."""

    def build():
        d, meta = gate_netlist(n_gates=gates, n_ff=max(64, gates * 2048 // 50_000), depth=40, seed=2)
        return sim.CompiledDesign(d.to_json(), meta.top), meta

    return _design(("netlist", gates), build)


def _crc32():
    def build():
        from rrtl_gb300.netlist import import_yosys_netlist

        with open(os.path.join(_ROOT, "tests", "golden", "crc32_gates.compact.json")) as f:
            c = json.load(f)
        y = {"modules": {c["top"]: {
            "ports": {k: {"direction": d, "bits": b} for k, (d, b) in c["ports"].items()},
            "cells": {f"c{i:04d}": {"type": t, "connections": n} for i, (t, n) in enumerate(c["cells"])}}}}
        return sim.CompiledDesign(import_yosys_netlist(y, c["top"]).to_json(), c["top"])

    return _design(("crc32",), build)


def _queue_jobs(case):
    """Sizes of the case's jobs: the same for every seed, which draws their stimulus."""
    rng = Rng(41)
    gates = [log_uniform_int(rng, 5_000, case["gates_hi"]) for _ in range(4)]
    return [(gates[i % 4], log_uniform_int(rng, 32, case["lanes_hi"]), log_uniform_int(rng, 20, case["cycles_hi"]),
             rng.uniform() < 0.3) for i in range(case["jobs"])]


# ------------------------------------------------------------------ prepare --
def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    s = {"kind": kind, "seed": seed}
    if kind == "tick":
        cd = _design(("counter",), lambda: sim.CompiledDesign(counter().to_json(), "Counter"))
        s["sim"] = sim.GpuBatchSimulator(cd, lanes=case["lanes"])
        s["en"] = rng.integers(0, 2, case["lanes"]).astype(np.uint32)
        s["rst"] = np.zeros(case["lanes"], dtype=np.uint32)
        v, m = s["sim"].snapshot_storage()  # every lane starts from a count of its own
        words = v.reshape(-1, case["lanes"])  # one word per signal
        words[cd.signal("count")[0]] = rng.integers(0, 256, case["lanes"])
        s["sim"].restore_storage(words.reshape(-1), m)
    elif kind == "counter":
        cd = _design(("counter",), lambda: sim.CompiledDesign(counter().to_json(), "Counter"))
        s["sim"] = sim.GpuBatchSimulator(cd, lanes=case["lanes"])
        s["args"] = dict(cycles=case["cycles"], seed=seed, record=["out"], mode=sim.REC_TRACE,
                         stim=[("clk", sim.STIM_CONST, 1), ("rst", sim.STIM_PULSE, 1), ("en", sim.STIM_RANDOM, 1)])
    elif kind == "cpu":
        cd = _design(("cpu",), lambda: sim.CompiledDesign(pipelined_cpu().to_json(), "Cpu8"))
        s["sim"] = sim.GpuBatchSimulator(cd, lanes=case["lanes"])
        s["sim"].set_memory_limbs("rom", cpu_rom_hashed(case["lanes"], seed=seed))
        s["args"] = dict(cycles=case["cycles"], seed=seed, record=["out_pc", "out_acc"], mode=sim.REC_HASH,
                         stim=[("clk", sim.STIM_CONST, 1), ("rst", sim.STIM_PULSE, 1)])
        s["limbs"] = ["out_pc", "out_acc"]
        s["mems"] = ["rf"]
    elif kind == "crc32":
        s["sim"] = sim.GpuBatchSimulator(_crc32(), lanes=case["lanes"])
        s["bits"] = [f"crc_{i}" for i in range(32)]
        s["args"] = dict(cycles=case["cycles"], seed=seed, record=s["bits"], mode=sim.REC_HASH,
                         stim=[("clk", sim.STIM_CONST, 1), ("rst", sim.STIM_PULSE, 1)]
                         + [(f"din_{i}", sim.STIM_RANDOM, i) for i in range(8)])
    elif kind == "netlist":
        cd, meta = _netlist(case["gates"])
        s["sim"] = sim.GpuBatchSimulator(cd, lanes=case["lanes"])
        stim, rec = netlist_run_spec(meta)
        s["args"] = dict(cycles=case["cycles"], seed=seed, record=rec, mode=sim.REC_HASH, stim=stim)
        if case["io"] == "state":
            s["bits"] = meta.regs
        else:
            s["args"]["mode"] |= sim.REC_TRACE
        if case["io"] == "replay":
            words = (case["lanes"] + 31) // 32
            s["args"]["input_trace"] = rng.integers(0, 1 << 32, (case["cycles"], len(meta.inputs), words),
                                                    dtype=np.uint32)
            s["args"]["stim"] = stim[:2] + [(p, sim.STIM_TRACE, i) for i, p in enumerate(meta.inputs)]
    elif kind == "fault":
        cd, meta = _netlist(case["gates"])
        s["sim"] = sim.GpuBatchSimulator(cd, lanes=case["lanes"])
        s["sim"].set_faults(job_faults(meta, case["lanes"], seed))
        stim, rec = netlist_run_spec(meta, uniform=True)
        s["args"] = dict(cycles=case["cycles"], seed=seed, record=rec, mode=sim.REC_HASH | sim.REC_DETECT, stim=stim)
    elif kind == "queue":
        s["ctx"] = sim.default_context()
        s["jobs"] = []
        for i, (gates, lanes, cycles, fault) in enumerate(_queue_jobs(case)):
            cd, meta = _netlist(gates)
            b = sim.GpuBatchSimulator(cd, lanes=lanes)
            if fault:
                b.set_faults(job_faults(meta, lanes, seed + i))
            stim, rec = netlist_run_spec(meta, uniform=fault)
            s["jobs"].append((b, dict(cycles=cycles, seed=seed + i, stim=stim, record=rec,
                                      mode=sim.REC_HASH | (sim.REC_DETECT if fault else 0))))
    elif kind == "bitslice":
        w = case["width"]
        cd = _design(("alu", w), lambda: sim.CompiledDesign(narrow_alu(w).to_json(), "Alu", bitslice=True))
        s["sim"] = sim.GpuBatchSimulator(cd, lanes=case["lanes"])
        s["bits"] = [f"acc[{p}]" for p in range(w)]
        s["args"] = dict(cycles=case["cycles"], seed=seed, record=[f"out[{p}]" for p in range(w)] + ["flag[0]"],
                         mode=sim.REC_HASH, stim=[("clk[0]", sim.STIM_CONST, 1), ("rst[0]", sim.STIM_PULSE, 1)]
                         + [(f"din[{p}]", sim.STIM_RANDOM, p) for p in range(w)]
                         + [(f"sel[{p}]", sim.STIM_RANDOM, 100 + p) for p in range(2)])
    else:
        n = case["instances"]
        js = _design(("fold", n), lambda: replicated_datapath(n).to_json())
        s["fold"] = sim.InstanceFoldSimulator(js, "Top", case["lanes"])
        s["sim"] = s["fold"].sim
        s["args"] = dict(cycles=case["cycles"], seed=seed, record=["o"], mode=sim.REC_TRACE,
                         stim=[("clk", sim.STIM_CONST, 1), ("rst", sim.STIM_PULSE, 1), ("din", sim.STIM_TRACE, 0)],
                         input_trace=rng.integers(0, 1 << 32, (case["cycles"], 1, n * case["lanes"]), dtype=np.uint32))
    return s


# ---------------------------------------------------------------------- run --
def _whole(a):
    """The same bits as signed integers, which torch can index (no copy)."""
    return a.view(np.int64 if a.dtype == np.uint64 else np.int32)


def run(s):
    kind = s["kind"]
    if kind == "tick":
        g = s["sim"]
        g.set_input("rst", s["rst"])
        g.set_input("en", s["en"])
        g.tick()
        return _whole(g.get_signal("count"))
    if kind == "queue":
        jobs = [s["ctx"].submit(b, **args) for b, args in s["jobs"]]
        s["ctx"].launch()
        s["ctx"].wait()
        return [[_whole(v) for v in (j.outputs["hash"], j.outputs["detect"]) if v is not None] for j in jobs]
    g = s["sim"]
    r = g.run(**s["args"])
    out = {k: _whole(v) for k, v in r.items() if v is not None}
    if "bits" in s:
        out["bits"] = _whole(g.get_signals_bits(s["bits"]))
    for name in s.get("limbs", ()):
        out[name] = _whole(g.get_signal_limbs(name))
    for name in s.get("mems", ()):
        out[name] = _whole(g.get_memory_limbs(name))
    return out


# --------------------------------------------------------------------- work --
def _netlist_work(gates, lanes, cycles, io="hash"):
    """Gate evaluations of whole 32-lane words (one bitwise operation each),
    and what must cross memory: lane state (flip-flops and inputs) in and
    out, recorded words out, trace words in."""
    words, ffs = (lanes + 31) // 32, max(64, gates * 2048 // 50_000)
    b = 2 * (ffs + 66) * words * 4 + cycles * 8
    if io == "state":
        b += ffs * words * 4
    if io in ("trace", "replay"):
        b += cycles * 64 * words * 4
    if io == "replay":
        b += cycles * 64 * words * 4
    return b, gates * words * cycles


def work(case):
    kind, lanes, cycles = case["kind"], case.get("lanes", 0), case.get("cycles", 1)
    words = (lanes + 31) // 32
    if kind == "tick":
        b, f = 4 * lanes * 5, 3 * lanes
    elif kind == "counter":
        b, f = 4 * lanes * (cycles + 10), 3 * lanes * cycles
    elif kind == "cpu":  # ROM, register file, data memory and 40 signal words per lane in, the written ones out
        b, f = 4 * lanes * (256 + 2 * (16 + 1024 + 40)) + 8 * cycles, 150 * lanes * cycles
    elif kind == "crc32":
        b, f = 4 * words * (2 * 42 + 32) + 8 * cycles, 195 * words * cycles
    elif kind == "netlist":
        b, f = _netlist_work(case["gates"], lanes, cycles, case["io"])
    elif kind == "fault":
        b, f = _netlist_work(case["gates"], lanes, cycles)
        b += lanes * 16
    elif kind == "queue":
        b = f = 0
        for gates, n, c, fault in _queue_jobs(case):
            x, y = _netlist_work(gates, n, c)
            b, f = b + x + (n * 16 if fault else 0), f + y
    elif kind == "bitslice":
        w = case["width"]
        b, f = 4 * words * 9 * w + 8 * cycles, 40 * w * words * cycles
    else:
        n = case["instances"] * lanes
        b, f = 4 * n * (2 * cycles + 10), 8 * n * cycles
    return {"bytes": b, "flops": f}


def exact(case, seed):
    return None
