"""The tests of test_gpu_parity.py on the pass kernels.

Meshes as small as theirs run as one resident launch by default; here every solver has
it switched off, so that the FP64 and FP32 gradient, face and cell passes, their launch
shapes and the level walk of the sequential time step are compared with the oracle too.
"""
import pytest

import test_gpu_parity
from supersonicflowsolver_b200.psst import Solver
from test_gpu_parity import (test_checkpoint_resumes_exactly, test_deterministic,  # noqa: F401
                             test_fp32_close_to_fp64_oracle, test_fp32_converged_field_close_to_fp64,
                             test_fp64_bit_exact_per_iteration, test_fp64_cell_limiters_match_oracle,
                             test_fp64_jacobi_local_time_matches_oracle, test_fp64_matches_reference_golden,
                             test_launch_shapes_and_autotune_keep_results, test_nonfinite_state_reports_error)

pytestmark = pytest.mark.gpu


class PassSolver(Solver):
    def __init__(self, *a, **kw):
        super().__init__(*a, **kw)
        self.use_wavefront(False)
        assert not self.schedule_info()["wavefront"]


@pytest.fixture(autouse=True)
def passes(monkeypatch):
    monkeypatch.setattr(test_gpu_parity, "Solver", PassSolver)
