"""bench.py names the stage kernels that a workload runs, and takes DRAM traffic and instruction mix only
from a capture of that kernel."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench


def test_captures_belong_to_the_kernel_that_runs():
    line = bench.stage_kernels("tgv_viscous_24_p5")
    assert line == ["line_kernel"]
    assert bench.ncu_traffic(line, 5, True, "fp64", 10)["bytes_per_launch"] > 0
    assert bench.measured_fp64_mix(line, 5, True, "fp64")["fp64_pipe_active"] > 0
    walls = ["periodic"] * 4 + ["wall"] * 2
    for kernels in (bench.stage_kernels("tgv_viscous_gl_24_p5"), bench.stage_kernels("tgv_viscous_24_p5", walls)):
        assert kernels != line
        assert bench.ncu_traffic(kernels, 5, True, "fp64", 10) is None
        assert bench.measured_fp64_mix(kernels, 5, True, "fp64") is None
    assert bench.stage_kernels("tgv_viscous_24_p5", walls) == ["line_kernel", "residual_kernel"]
    assert bench.stage_kernels("tgv_viscous_24_p5", ["periodic"] * 6) == line
