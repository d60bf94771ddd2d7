"""The rules that choose how a box is looked up, at the sizes where they turn:
x boxes about 16, 17 (the widest one lookup holds) and 32 cells (the widest a
fused row takes), tall y boxes, rows that end inside a word, obstacles (the
valid-cell test), several rows of representatives.  Bit-exact against the
oracle, both methods, both loops."""
import ctypes

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


def box_case(shape, cells, inputs, obstacle):
    """Disturbances of cells[d] / 2 grid cells: boxes of about cells[d] + 1."""
    c = C.unicycle_grid_case(shape, inputs, "box_%dx%dx%dx%d" % shape, max_iterations=64)
    c["disturbance_half_width"] = [cells[d] / 2.0 * c["state_eta"][d] for d in range(4)]
    c["constraint"] = "none"
    c["candidate_ellipse"] = [0.0, 0.0, 1.0, 1.0, 2.5]
    if obstacle:
        c["obstacles"] = [[0.9, 0.9, c["state_lb"][2], c["state_lb"][3], 1.2, 1.2, c["state_ub"][2], c["state_ub"][3]]]
        c["constraint"] = "quadric"   # the valid set is not the safe set
        c["constraint_params"] = [1.0, 1.0, 3.0, 1.9]
    return c


@pytest.mark.parametrize("obstacle", [False, True], ids=["free", "obstacle"])
@pytest.mark.parametrize("shape,cells,inputs", [
    ((33, 9, 5, 3), (0.0, 0.0, 0.0, 0.0), (3, 3)),      # narrow boxes, a row one cell past a word
    ((63, 20, 6, 4), (14.5, 1.0, 0.0, 0.0), (3, 3)),    # x boxes of 15 to 17 cells
    ((64, 20, 6, 4), (16.5, 1.0, 0.0, 0.0), (3, 3)),    # 17 to 18
    ((95, 40, 5, 3), (30.2, 3.0, 1.0, 0.0), (3, 3)),    # 31 to 32
    ((96, 12, 5, 3), (34.0, 0.0, 0.0, 0.0), (3, 3)),    # beyond a word: prefix counts
    ((31, 64, 4, 3), (0.0, 29.5, 0.0, 0.0), (3, 3)),    # y boxes to 32 rows
    ((250, 7, 8, 5), (4.0, 0.0, 1.0, 1.0), (5, 5)),     # eight words a row
    ((257, 7, 8, 5), (4.0, 0.0, 1.0, 1.0), (5, 5)),     # wide grid, box table
    ((24, 24, 12, 8), (0.0, 0.0, 0.0, 0.0), (21, 17)),  # more inputs than a pass of representatives
])
def test_box_lookups_against_oracle(ctx, shape, cells, inputs, obstacle):
    case = box_case(shape, cells, inputs, obstacle)
    want = O.solve(case)
    solved = 0
    for method in (G.METHOD_AUTO, G.METHOD_STORED, G.METHOD_FUSED):
        absn = G.Abstraction(ctx, case)
        try:
            p = G.Problem(ctx, absn, case, method)
        except G.GscError as e:
            assert method == G.METHOD_FUSED and e.status == 4, e
            absn.close()
            continue
        for graph in (False, True):
            p.solve(graph=graph)
            got = p.read()
            assert_same_result(got, want, f"{case['name']}/{method}/graph={graph}")
            assert got["iterations"] == want["iterations"] and got["message"] == want["message"]
            solved += 1
        p.close()
        absn.close()
    assert solved >= 4


@pytest.mark.parametrize("shape", [(33, 9, 5, 3), (1, 9, 8, 3), (9, 1, 8, 3), (33, 5, 1, 3), (17, 6, 8, 1),
                                   (64, 20, 6, 4)])
def test_noalloc_corner_tests_against_oracle(ctx, shape):
    """Corner cells before counts over the caller's pairs, and extents of one
    cell (whose division is none)."""
    import torch
    case = box_case(shape, (1.5, 1.0, 1.0, 0.0), (5, 5), False)
    want = O.solve(case)
    absn = G.Abstraction(ctx, case)
    p = G.Problem(ctx, absn, case, G.METHOD_AUTO)
    pairs = [np.ascontiguousarray(a) for a in p.export_abstraction()]
    p.close()
    absn.close()
    dev = [torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a.view(np.uint8)).cuda() for a in
           pairs + [np.asarray(want["valid_mask"]), np.asarray(want["candidate_mask"])]]
    S = int(np.prod(shape))
    out = [torch.empty(S, dtype=torch.uint8, device="cuda"), torch.empty(S, dtype=torch.int32, device="cuda"),
           torch.empty(S, dtype=torch.int32, device="cuda")]
    st = G.lib().gsc_fixpoint_noalloc((ctypes.c_uint32 * 4)(*shape), pairs[0].size // S, 2,
                                      *[ctypes.c_void_p(t.data_ptr()) for t in dev], case["max_iterations"],
                                      *[ctypes.c_void_p(t.data_ptr()) for t in out], None,
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    torch.cuda.synchronize()
    for got, name in zip(out, ("reachable_mask", "controller", "reach_step")):
        w = np.asarray(want[name])
        assert np.array_equal(got.cpu().numpy().view(w.dtype), w), name
