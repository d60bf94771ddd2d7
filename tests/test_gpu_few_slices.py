"""Grids of few (theta, v) slices, where a slice's rows are shared by several
blocks: row counts about a block's, rows of one to eight words, one slice to
more than 300 (where a slice is one block's again), with and without obstacles,
one and several substeps.  Bit-exact against the oracle, both loops."""
import numpy as np
import pytest

import gsc_b200 as G
import gsc_cases as C
import oracle as O
from helpers import assert_same_result

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = G.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("obstacle", [False, True], ids=["free", "obstacle"])
@pytest.mark.parametrize("shape,inputs,substeps,tau", [
    ((40, 257, 4, 3), (5, 5), 1, 0.1),      # twelve slices, a row past 16 blocks
    ((9, 1000, 3, 2), (7, 7), 1, 0.05),     # six
    ((33, 400, 1, 1), (9, 9), 4, 0.02),     # one
    ((256, 33, 6, 3), (5, 5), 1, 0.1),      # eight words a row
    ((70, 48, 16, 9), (5, 5), 2, 0.1),      # 144: two blocks a slice
    ((70, 47, 20, 15), (6, 6), 1, 0.1),     # 300
    ((70, 48, 43, 7), (5, 5), 1, 0.1),      # 301: one
])
def test_rows_of_a_slice_in_several_blocks(ctx, shape, inputs, substeps, tau, obstacle):
    case = C.unicycle_grid_case(shape, inputs, "few_%dx%dx%dx%d" % shape, max_iterations=48)
    case.update(integration_substeps=substeps, sample_time=tau, disturbance_half_width=[0.005] * 4)
    if obstacle:
        case["obstacles"] = [[0.9, 0.9, case["state_lb"][2], case["state_lb"][3], 1.3, 1.2, case["state_ub"][2],
                              case["state_ub"][3]]]
    want = O.solve(case)
    absn = G.Abstraction(ctx, case)
    p = G.Problem(ctx, absn, case, G.METHOD_AUTO)
    for graph in (False, True):
        p.solve(graph=graph)
        got = p.read()
        assert_same_result(got, want, f"{case['name']}/graph={graph}")
        assert got["iterations"] == want["iterations"] and got["message"] == want["message"]
    p.close()
    absn.close()
