"""The flat gate program run on the CPU as the flat kernel decodes it
(tests/native/flat_program_emu.cpp): per-warp entry streams with their level
barriers, packed cells, registers folded into the levels and the commit list.
The emulator checks what the kernel relies on unchecked (equal barriers on
every warp, no row read or written in the level another lane writes it) and
its per-cycle output hash must equal the bit-parallel oracle's."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import binding as ob
from rrtl_gb300 import sim
from rrtl_gb300.workloads import gate_netlist, narrow_alu, netlist_run_spec

from .helpers import crc32_netlist_json, oracle_bp_run
from .test_gate_program_emu import _register_mix

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC = [os.path.join(HERE, "native", "flat_program_emu.cpp")] + [
    os.path.join(ROOT, "rrtl_gb300", "csrc", f) for f in ("flatprog.cpp", "gateprog.cpp", "design.cpp", "lower.cpp")]
LIB = os.path.join(HERE, "native", "_build", "libflat_emu.so")
P, U32, U64 = ctypes.POINTER, ctypes.c_uint32, ctypes.c_uint64


@pytest.fixture(scope="module")
def emu():
    deps = SRC + [os.path.join(ROOT, "rrtl_gb300", "csrc", h) for h in
                  ("flatprog.h", "flat_shape.h", "gateprog.h", "design.h", "lower.h", "json.h", "stim.h")]
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < max(os.path.getmtime(p) for p in deps):
        os.makedirs(os.path.dirname(LIB), exist_ok=True)
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", LIB + ".tmp"] + SRC, check=True)
        os.replace(LIB + ".tmp", LIB)
    L = ctypes.CDLL(LIB)
    L.emu_flat_run.argtypes = [ctypes.c_char_p, ctypes.c_size_t, ctypes.c_char_p, U32, U32, U32, U32, U32, U32, U64,
                               U64, U64, U32, P(U32), P(U32), P(U64), U32, P(U32), P(U64), P(U32), ctypes.c_char_p,
                               ctypes.c_size_t]
    return L


STATS = ("two", "three", "levels", "slots", "entries", "wavefronts", "floor", "commit")


def _emulate(L, js, top, od, stim, rec, lanes, cycles, seed, V, pack=1, fold=1, warps=16, max_slots=0, lane_base=0):
    arr = lambda v, t: np.ascontiguousarray(v, dtype=t)
    sig, kind = arr([od.signal(n) for n, _, _ in stim], np.uint32), arr([k for _, k, _ in stim], np.uint32)
    param, rsig = arr([p for _, _, p in stim], np.uint64), arr([od.signal(r) for r in rec], np.uint32)
    out, stats, err = np.zeros(cycles, dtype=np.uint64), np.zeros(16, dtype=np.uint32), ctypes.create_string_buffer(512)
    ptr = lambda a, t: a.ctypes.data_as(P(t))
    raw = js.encode()
    rc = L.emu_flat_run(raw, len(raw), top.encode(), V, pack, fold, warps, max_slots, lanes, cycles, seed, lane_base,
                        len(sig), ptr(sig, U32), ptr(kind, U32), ptr(param, U64), len(rsig), ptr(rsig, U32),
                        ptr(out, U64), ptr(stats, U32), err, len(err))
    assert rc == 0, err.value.decode()
    return out, dict(zip(STATS, stats.tolist()))


def _oracle(od, stim, rec, lanes, cycles, seed, lane_base=0):
    return oracle_bp_run(od, lanes, cycles, seed, [(od.signal(n), k, p) for n, k, p in stim],
                         [od.signal(r) for r in rec], 2, lane_base=lane_base)["hash"]


@pytest.fixture(scope="module")
def netlist():
    d, meta = gate_netlist(n_gates=6000, n_ff=256, n_pi=24, n_po=24, depth=14, seed=31)
    js = d.to_json()
    return js, meta, ob.OracleDesign(js, meta.top)


@pytest.mark.parametrize("V,warps", [(4, 16), (4, 8), (2, 16), (1, 16), (2, 24), (1, 24)])
@pytest.mark.parametrize("pack,fold", [(0, 0), (1, 0), (0, 1), (1, 1), (2, 1)])
def test_netlist_equals_the_oracle(emu, netlist, V, warps, pack, fold):
    js, meta, od = netlist
    stim, rec = netlist_run_spec(meta)
    h, st = _emulate(emu, js, meta.top, od, stim, rec, 100, 12, 41, V, pack, fold, warps)
    assert np.array_equal(h, _oracle(od, stim, rec, 100, 12, 41))
    assert st["commit"] < 256 if fold else st["commit"] == 256
    # rows read and written near one wavefront per group and position
    assert st["floor"] <= st["wavefronts"] <= 1.10 * st["floor"], st


@pytest.mark.parametrize("blocks", [1, 2, 7, 152])
def test_split_tiles_cover_a_run_once(emu, blocks):
    """Tiles past one a block (fewer: one launch of whole tiles), the shortest runs and the longest."""
    emu.emu_flat_parts.argtypes = [U32, U64, U32]
    for tiles in [blocks, blocks + 1, blocks + 3, 2 * blocks - 1, 2 * blocks, 3 * blocks + 1, 2048]:
        for cycles in [4, 5, 7, 100, 2**32 - 1]:
            if tiles >= blocks:
                assert emu.emu_flat_parts(tiles, cycles, blocks) == 0, (tiles, cycles)


@pytest.mark.parametrize("V", [4, 2, 1])
def test_closing_settle_writes_every_signal_back(emu, netlist, V):
    """The settle's program alone, its write-backs and the source rows standing for every net."""
    js, meta, od = netlist
    stim, rec = netlist_run_spec(meta)
    rec = list(dict.fromkeys(rec + meta.gate_names))
    h, st = _emulate(emu, js, meta.top, od, stim, rec, 40, 6, 17, V, pack=3)
    assert np.array_equal(h, _oracle(od, stim, rec, 40, 6, 17))
    d, top, outs = _register_mix()
    js = d.to_json()
    od = ob.OracleDesign(js, top)
    stim = [("clk", sim.STIM_CONST, 1), ("rst", sim.STIM_PULSE, 3), ("rstn", sim.STIM_RANDOM, 9),
            ("a", sim.STIM_RANDOM, 1), ("b", sim.STIM_RANDOM, 2), ("c", sim.STIM_RANDOM, 3)]
    h, _ = _emulate(emu, js, top, od, stim, outs, 70, 20, 13, V, pack=3)
    assert np.array_equal(h, _oracle(od, stim, outs, 70, 20, 13))


def test_a_shorter_slot_array_keeps_the_results(emu, netlist):
    js, meta, od = netlist
    stim, rec = netlist_run_spec(meta)
    _, free = _emulate(emu, js, meta.top, od, stim, rec, 40, 1, 3, 4)
    cap = free["slots"] - 1
    h, st = _emulate(emu, js, meta.top, od, stim, rec, 40, 8, 3, 4, max_slots=cap - cap // 50)
    assert st["slots"] < free["slots"]
    assert np.array_equal(h, _oracle(od, stim, rec, 40, 8, 3))


@pytest.mark.parametrize("V", [4, 1])
def test_register_forms_equal_the_oracle(emu, V):
    d, top, outs = _register_mix()
    js = d.to_json()
    od = ob.OracleDesign(js, top)
    stim = [("clk", sim.STIM_CONST, 1), ("rst", sim.STIM_PULSE, 3), ("rstn", sim.STIM_RANDOM, 9),
            ("a", sim.STIM_RANDOM, 1), ("b", sim.STIM_RANDOM, 2), ("c", sim.STIM_RANDOM, 3)]
    h, _ = _emulate(emu, js, top, od, stim, outs, 70, 40, 13, V)
    assert np.array_equal(h, _oracle(od, stim, outs, 70, 40, 13))


@pytest.mark.parametrize("V", [4, 2])
def test_shift_chain_and_random_register_graphs(emu, V):
    """Registers fed by registers: a chain longer than the levels (its tail
    stays on the commit list), swaps, self loops, shared and constant D nets."""
    from rrtl_gb300.builder import Design, lit_u, mux, uint
    from rrtl_gb300.workloads import Rng

    for seed in range(12):
        rng = Rng(seed)
        d = Design()
        m = d.module("R")
        clk, rst = m.input("clk", uint(1)), m.input("rst", uint(1))
        ins = [m.input(f"i{k}", uint(1)) for k in range(3)]
        regs = [m.reg(f"r{k}", uint(1)) for k in range(14)]
        pool = list(ins) + list(regs)
        wires = []
        for k in range(rng.below(20)):
            a, b, c = (pool[rng.below(len(pool))] for _ in range(3))
            e = [a & b, a | b, a ^ b, ~(a & b), mux(a, b, c), ~a.value()][rng.below(6)]
            w = m.wire(f"w{k}", uint(1))
            m.assign(w, e)
            pool.append(w)
            wires.append(w)
        for k, r in enumerate(regs):
            m.clock(r, clk)
            if rng.below(2):
                m.reset(r, rst, rng.below(2))
            pick = rng.below(8)
            if k and pick < 4:
                m.next(r, regs[k - 1])  # chain
            elif pick == 4:
                m.next(r, ~r.value())
            elif pick == 5:
                m.next(r, lit_u(rng.below(2), 1))
            else:
                m.next(r, pool[rng.below(len(pool))] ^ pool[rng.below(len(pool))])
        outs = []
        for k in range(5):
            o = m.output(f"o{k}", uint(1))
            m.assign(o, pool[rng.below(len(pool))])
            outs.append(f"o{k}")
        js = d.to_json()
        od = ob.OracleDesign(js, "R")
        stim = [("clk", sim.STIM_CONST, 1), ("rst", sim.STIM_PULSE, 2)] + [(f"i{k}", sim.STIM_RANDOM, k) for k in range(3)]
        h, _ = _emulate(emu, js, "R", od, stim, outs, 40, 25, seed, V)
        assert np.array_equal(h, _oracle(od, stim, outs, 40, 25, seed)), seed


def test_crc32_and_plane_design_equal_the_oracle(emu):
    js = crc32_netlist_json().to_json()
    od = ob.OracleDesign(js, "crc32")
    stim = [("clk", sim.STIM_CONST, 1), ("rst", sim.STIM_PULSE, 1)] + [(f"din_{i}", sim.STIM_RANDOM, i) for i in range(8)]
    rec = [f"crc_{i}" for i in range(32)]
    for base in (0, 4096):
        h, _ = _emulate(emu, js, "crc32", od, stim, rec, 100, 20, 7, 4, lane_base=base)
        assert np.array_equal(h, _oracle(od, stim, rec, 100, 20, 7, base)), base
    js = sim.bitslice_json(narrow_alu(9), "Alu")
    od = ob.OracleDesign(js, "Alu")
    stim = [("clk[0]", sim.STIM_CONST, 1), ("rst[0]", sim.STIM_PULSE, 1)]
    stim += [(f"din[{p}]", sim.STIM_RANDOM, p) for p in range(9)] + [(f"sel[{p}]", sim.STIM_RANDOM, 50 + p) for p in range(2)]
    rec = [f"out[{p}]" for p in range(9)] + ["flag[0]"]
    h, _ = _emulate(emu, js, "Alu", od, stim, rec, 33, 30, 5, 2)
    assert np.array_equal(h, _oracle(od, stim, rec, 33, 30, 5))
