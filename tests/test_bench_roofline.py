"""The roofline fields of bench.py's plain FP64 M2L: the work the kernel that runs cannot do without, never more than
the pipe's peak at measured times."""
import os
import sys

import pytest

from conftest import ROOT

sys.path.insert(0, ROOT)
import bench  # noqa: E402


# flops as the library counts them (2 P^2 a pair) and kernel times measured on a B200
@pytest.mark.parametrize("workload,tflop,ms,kernel", [("c3", 21.8, 284.0, "k_m2l_sym"), ("c4", 0.62, 9.4, "k_m2l_sym"),
                                                      ("c2", 0.018, 1.1, "k_m2l_f64")])
def test_fp64_roofline_is_of_the_kernel_that_runs(workload, tflop, ms, kernel):
    roof = bench.fp64_m2l_roof(bench.WORKLOADS[workload], tflop * 1e12, ms)
    assert roof["kernel"].startswith(kernel)
    assert 0.0 < roof["frac"] <= 1.0
    assert bench.fp64_m2l_roof(bench.WORKLOADS[workload], tflop * 1e12, 0.0)["achieved"] is None
