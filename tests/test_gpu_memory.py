"""Device memory of a fused query: bounded by its sets, tables and copies with
nothing beside them, so that budgets sized by that keep admitting it; and where
the dilated copies do not fit, D' is read without them, to the same result."""
import numpy as np
import pytest

import gsc_b200 as G
import gsc_cases as C
import oracle as O
from helpers import assert_same_result

pytestmark = pytest.mark.gpu


def bound(case, problem_widths, need_valid):
    """Bytes of: masks and results (15 a state, with the lowest input found so
    far), eight bit-sliced sets, per-axis boxes, classes and representatives a
    (slice, input), one dilated copy a pair of box widths, and per-cell tables."""
    n, m = C.grid_shape(case)
    S, M = int(np.prod(n)), m[0] * m[1]
    slices, W = n[2] * n[3], (n[0] + 31) // 32
    planes, words = slices * M, slices * n[1] * W
    classes = 4 + 9 * W if case["integration_substeps"] == 1 else (4 + 9 * W + 3) // 4 * 4
    copies = problem_widths * words * (2 if need_valid else 1)
    safe = n[0] * n[1] if case["constraint"] != "none" else 0
    return (15 * S + 4 * (8 * words + copies) + planes * (4 * (n[0] + n[1]) + 4 * classes + 1) + safe +
            64 * len(case["obstacles"]) + 8 * (slices * ((n[1] + 31) // 32) + 1) + 8 * (n[2] * m[1] + n[3] * m[0]) +
            32 * (case["max_iterations"] + 2) + 1024)


def obstacles(case):
    c = C.clone(case)
    c["obstacles"] = [[1.2, 1.2, c["state_lb"][2], c["state_lb"][3], 1.6, 1.6, c["state_ub"][2], c["state_ub"][3]]]
    return c


def hyperbolic(n, m):
    c = C.hyperbolic_demo_case()
    c["state_eta"] = [(u - lo) / k for lo, u, k in zip(c["state_lb"], c["state_ub"], n)]
    c["input_eta"] = [(u - lo) / k for lo, u, k in zip(c["input_lb"], c["input_ub"], m)]
    return c


CASES = [
    C.unicycle_grid_case((24, 24, 16, 8), (50, 50)), C.unicycle_grid_case((16, 16, 12, 6), (250, 16)),
    C.small_case(), obstacles(C.small_case()), C.unicycle_grid_case((24, 24, 12, 8), (21, 17)),
    obstacles(C.unicycle_grid_case((24, 24, 12, 8), (21, 17))), obstacles(C.unicycle_grid_case((16, 16, 16, 16), (10, 10))),
    obstacles(C.unicycle_grid_case((17, 130, 9, 5), (3, 3))), hyperbolic((40, 40, 20, 8), (5, 5)),
    obstacles(hyperbolic((35, 35, 32, 7), (5, 5))), C.default_case(),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, C.grid_shape(c)[0] + C.grid_shape(c)[1])))
def test_fused_query_stays_within_its_bound(case):
    with G.Context(0) as c:
        a = G.Abstraction(c, case)
        p = G.Problem(c, a, case, G.METHOD_FUSED)
        used = p.timings()["device_bytes"]
        assert used <= bound(case, 1, bool(case["obstacles"])), used
        p.close()
        a.close()


def test_without_room_for_the_dilated_copies():
    """Budgets a little below what the query takes otherwise: fewer launches an
    iteration, the same result."""
    case = obstacles(hyperbolic((48, 40, 31, 12), (8, 8)))
    case["max_iterations"] = 4
    want = O.solve(case)
    with G.Context(0) as c:
        c.set_memory_budget((64 << 20) - 1)   # below a full-size region of the pool
        a = G.Abstraction(c, case)
        held = c.memory_in_use()
        p = G.Problem(c, a, case, G.METHOD_FUSED)
        p.solve()
        most = p.timings()
        assert_same_result(p.read(), want, "with copies")
        full = c.memory_in_use() - held
        p.close()
        c.trim()
        seen = set()
        for share in (0.99, 0.98, 0.97, 0.96, 0.95, 0.93, 0.5):
            c.set_memory_budget(held + int(full * share))
            try:
                p = G.Problem(c, a, case, G.METHOD_FUSED)
            except G.GscError as e:
                assert e.status == 3
                seen.add("refused")
                c.trim()
                continue
            p.solve(graph=True)
            p.solve()
            t = p.timings()
            seen.add(t["kernel_launches"] < most["kernel_launches"])
            got = p.read()
            assert_same_result(got, want, f"{share} of the memory")
            assert got["iterations"] == want["iterations"] and got["message"] == want["message"]
            p.close()
            c.trim()
        a.close()
    assert True in seen and "refused" in seen, seen
