"""Grids whose slices have more representative inputs than the satisfaction
kernel takes at a time (256, fewer where a slice has more than 128 rows), with
states that only an input of a later pass satisfies.  Bit-exact against the
oracle, through both loops and in a batch."""
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


def steering_case(shape, inputs, T, accel, omega, ymax, obstacle=False, **over):
    """32 substeps of strong inputs: each moves the successor to other cells."""
    c = C.unicycle_grid_case(shape, inputs, "steering_%dx%dx%dx%d" % shape, max_iterations=24)
    c.update(sample_time=T, integration_substeps=32, input_lb=[-accel, -omega], input_ub=[accel, omega],
             input_eta=[2 * accel / inputs[0], 2 * omega / inputs[1]], disturbance_half_width=[0.0] * 4,
             constraint_params=[1.0, 1.0, 9.0, ymax], candidate_ellipse=[0.0, -0.9, 1.0, 1.0, 0.8])
    if obstacle:   # valid is less than safe
        c["obstacles"] = [[0.4, 0.1, c["state_lb"][2], c["state_lb"][3], 1.1, 0.6, c["state_ub"][2], c["state_ub"][3]]]
    c.update(over)
    return C.checked(c)


CASES = {
    "256": lambda: steering_case((8, 128, 12, 4), (8, 56), 1.0, 0.4, 3.1, 1.9),
    "128_obstacle": lambda: steering_case((8, 256, 12, 4), (8, 32), 0.5, 0.8, 6.2, 1.9, obstacle=True),
    "31": lambda: steering_case((6, 1056, 12, 4), (6, 40), 0.02, 10.0, 150.0, 1.3,
                                candidate_ellipse=[0.0, 0.0, 1.0, 1.0, 0.64],
                                disturbance_half_width=[0.01, 0.05, 0.01, 0.01]),
}


def passes(case):
    """Most distinct inputs of a slice (by their pairs: at most as many as its
    representatives) and the representatives of a pass; states per slice whose
    controller comes after a pass of distinct inputs, most of a slice."""
    (n0, n1, n2, n3), m = C.grid_shape(case)
    M = m[0] * m[1]
    mn, mx, ok = (a.reshape(n2 * n3, n0 * n1, M).astype(np.uint64) for a in O.abstraction(case))
    mix = np.random.default_rng(1).integers(1, 2**63, size=(n0 * n1, 1), dtype=np.uint64)
    key = ((mn * np.uint64(1000003) + mx * np.uint64(2) + ok) * mix).sum(axis=1)
    first = [np.sort(np.unique(k, return_index=True)[1]) for k in key]
    return first, min(256, 1024 // ((n1 + 31) // 32))


@pytest.fixture(scope="module")
def solved():
    out = {}
    for name, make in CASES.items():
        case = make()
        want = O.solve(case)
        first, per_pass = passes(case)
        assert max(len(f) for f in first) > per_pass
        ctl = np.asarray(want["controller"]).reshape(len(first), -1)
        late = [np.count_nonzero(c[c != 0xFFFFFFFF] >= f[per_pass]) if len(f) > per_pass else 0
                for c, f in zip(ctl, first)]
        assert max(late) > 100, late
        out[name] = (case, want)
    return out


def check(got, want, label):
    assert_same_result(got, want, label)
    for k in ("iterations", "message", "reachable_states", "certified_candidates"):
        assert got[k] == want[k], (label, k)


@pytest.mark.parametrize("name", sorted(CASES))
def test_solves_against_oracle(ctx, solved, name):
    case, want = solved[name]
    absn = G.Abstraction(ctx, case)
    p = G.Problem(ctx, absn, case, G.METHOD_FUSED)
    for graph in (False, True):
        p.solve(graph=graph)
        check(p.read(), want, f"{name}/graph={graph}")
    p.close()
    absn.close()


@pytest.mark.parametrize("warp", [False, True], ids=["block", "warp"])
def test_batch_against_oracle(ctx, solved, warp):
    names = sorted(CASES)
    b = G.Batch(ctx, [solved[n][0] for n in names], sat_threads=64, sat_warp_tasks=warp)
    b.solve(graph=True)
    for i, n in enumerate(names):
        check(b.read(i), solved[n][1], f"batch/{n}")
    b.close()
