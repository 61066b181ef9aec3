"""A run's stimulus and record tables as make_run lays them out (no device)."""
import numpy as np
import pytest

from rrtl_gb300 import sim


@pytest.fixture(scope="module")
def shape():
    cd = object.__new__(sim.CompiledDesign)
    cd.h, cd._cache, cd._engine = None, {"a": (0, 1, 0), "b": (1, 1, 0), "c": (2, 1, 1)}, sim.ENGINE_GATE
    cd.signal = lambda name: cd._cache[name]
    return sim._RunShape(cd, 64)


def _stim(run):
    return [(run.stim[i].signal, run.stim[i].kind, run.stim[i].param) for i in range(run.n_stim)]


@pytest.mark.parametrize("t", [int, np.int64, np.int32, np.uint64, np.uint32, np.uint8, np.int8])
def test_stimulus_takes_any_integer(shape, t):
    r = shape.make_run(4, stim=[("a", t(sim.STIM_PULSE), t(5)), (1, t(sim.STIM_CONST), t(1))])
    assert _stim(r) == [(0, sim.STIM_PULSE, 5), (1, sim.STIM_CONST, 1)]


def test_stimulus_parameters_fill_their_field(shape):
    ps = [(2**64 - 1, 2**64 - 1), (-1, 2**64 - 1), (np.int64(-1), 2**64 - 1), (np.uint64(2**63), 2**63),
          (2**64 + 3, 3), (True, 1)]
    r = shape.make_run(4, stim=[("b", sim.STIM_RANDOM, p) for p, _ in ps])
    assert _stim(r) == [(1, sim.STIM_RANDOM, want) for _, want in ps]


@pytest.mark.parametrize("bad", [1.5, None, "1", np.float64(2)])
def test_stimulus_of_other_types_is_refused(shape, bad):
    for entry in (("a", sim.STIM_CONST, bad), ("a", bad, 1), (bad if bad != "1" else 1.0, sim.STIM_CONST, 1)):
        with pytest.raises(TypeError):
            shape.make_run(4, stim=[entry])


@pytest.mark.parametrize("n", [2, 4])
def test_stimulus_entries_have_three_values(shape, n):
    with pytest.raises(ValueError):
        shape.make_run(4, stim=[("a", sim.STIM_CONST, 1), ("b", sim.STIM_CONST, 1, 0)[:n]])


@pytest.mark.parametrize("bad", [2**32, 2**32 + 1, -1])
def test_indices_outside_32_bits_are_refused(shape, bad):
    with pytest.raises(OverflowError):
        shape.make_run(4, record=["a", bad])
    with pytest.raises(OverflowError):
        shape.design.indices([bad])


def test_records_by_name_and_index(shape):
    r = shape.make_run(4, record=["c", 1, "a"])
    assert [r.record[i] for i in range(r.n_record)] == [2, 1, 0]
    assert shape.make_run(4).n_stim == 0 and shape.make_run(4).n_record == 0
