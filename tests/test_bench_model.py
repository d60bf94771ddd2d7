"""bench.py's account of the satisfaction kernel: the kernel that a solve runs,
the bytes it must move, and the committed counters of it."""
import importlib.util
import os

import pytest

import gsc_cases as C
from helpers import ROOT


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(ROOT, "bench.py"))
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module


def test_kernel_of_a_solve(bench):
    assert bench.satisfaction_kernel(2, (65, 65, 38, 25), 1) == "k_slice"
    assert bench.satisfaction_kernel(1, (65, 65, 38, 25), 1) == "k_sat_bits"
    assert bench.satisfaction_kernel(1, (300, 24, 20, 8), 1) == "k_sat_bits"
    assert bench.satisfaction_kernel(1, (65, 65, 38, 25), 2) == "k_sat_stored"
    assert bench.satisfaction_kernel(1, (300, 24, 20, 8), 4) == "k_sat_stored_wide"


def test_bytes_a_launch_must_move(bench):
    t = {"sat_launches": 10, "aux_count": 400, "pair_tests": 10000}
    # 38 * 25 slices of 65 rows of three words, padded to four: active and D' once, 40 records a launch
    assert bench.algorithmic_bytes("k_slice", (65, 65, 38, 25), t) == 8 * 950 * 196 + 32 * 40
    assert bench.algorithmic_bytes("k_sat_bits", (300, 24, 20, 8), t) == 8 * 1000 + 7 * 300 * 24 * 20 * 8
    assert bench.algorithmic_bytes("k_sat_stored_wide", (300, 24, 20, 8), t) == 16 * 1000 + 7 * 300 * 24 * 20 * 8


def test_committed_figures_of_the_current_kernels(bench):
    workload = C.demo_scale_case()["name"]
    traffic = bench.ncu_traffic("k_slice", workload)
    assert traffic and 1e5 < traffic < 1e9
    issue = bench.issue_roofline("k_slice", workload, 0.02, 1965.0, 148)
    assert issue and 0 < issue["frac"] < 1
    assert bench.ncu_traffic("k_sat_bits", C.serve_mid_case()["name"]) > 1e8
