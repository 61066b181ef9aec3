"""The fused kernels over many cycles: runs that the flat kernel would take,
kept off it (RRTL_FLAT=0), by the same checks against the oracle. The fused
kernels still run what the flat one does not take: runs of under four cycles,
programs that do not fit its rows, fault runs that drive a register, serving."""
import pytest

from . import test_gpu_gate as gate, test_gpu_queue as queue
from .test_gpu_gate import small_netlist  # noqa: F401  (fixtures of the shared checks)
from .test_gpu_gate_jit import test_faults_and_explicit_widths_use_the_fused_kernel  # noqa: F401
from .test_gpu_queue import designs  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def fused_kernels(monkeypatch):
    monkeypatch.setenv("RRTL_FLAT", "0")


test_tile_widths_match_the_oracle = gate.test_netlist_tile_widths_match_oracle
test_faults_at_tile_widths_match_the_oracle = gate.test_netlist_faults_tile_widths_match_oracle
test_faults_match_the_oracle = gate.test_netlist_faults_match_oracle
test_design_compiled_kernel_equals_the_generic_one = gate.test_design_compiled_fused_kernel_equals_generic
test_narrow_tiles_of_a_large_netlist = gate.test_large_netlist_runs_fused_at_narrow_tiles
test_full_size_netlist_equals_the_plain_path = gate.test_full_size_netlist_fused_equals_plain
test_state_after_ticks_matches_the_oracle = gate.test_tick_many_and_snapshot_match_oracle
test_queued_jobs_equal_runs_alone = queue.test_queue_jobs_match_runs_alone
test_queued_jobs_match_the_oracle = queue.test_queue_job_matches_oracle
test_queued_fault_jobs_match_the_oracle = queue.test_queue_fault_job_detection_matches_oracle
