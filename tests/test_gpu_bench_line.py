"""bench.py describes the kernels that its timed region runs."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("workload,resident", [("ramp2d_120x40_fp64", True), ("wedge3d_750k_tets", False)])
def test_line_names_the_form_that_ran(workload, resident):
    out = subprocess.run([sys.executable, "bench.py", "--workload", workload, "--steps", "6", "--warmup", "3",
                          "--no-cpu-baseline"], cwd=ROOT, check=True, capture_output=True, text=True).stdout
    line = json.loads(out.strip().splitlines()[-1])
    assert line["finite"] and line["value"] > 0
    kernels = set(line["kernel_ms_per_iteration"])
    if resident:
        assert line["gpu_launches"] == 1
        assert line["roofline"]["kernel"] == "resident" and kernels == {"resident"}
        assert abs(line["kernel_ms_per_iteration"]["resident"] - line["ms_per_step"]) < 1e-6 * line["ms_per_step"]
    else:
        assert line["gpu_launches"] >= 6 * 10 and {"gradient", "face", "cell"} <= kernels
        assert line["roofline"]["kernel"] in kernels
    assert line["config"]["cuda_graphs"] == (not resident)
