"""What a query is refused for when device memory is short: a candidate set
with invalid states is reported as such wherever the masks and per-axis boxes
fit the budget, and as a lack of memory only where they do not."""
import numpy as np
import pytest

import gsc_b200 as G
import gsc_cases as C

pytestmark = pytest.mark.gpu


def rounded(n):
    return (max(int(n), 1) + 255) // 256 * 256


def judged_bytes(case, fused):
    """Device memory of the buffers that judge a query: masks, counters,
    per-axis boxes, plan record, and with the fused method its plane classes."""
    n, m = C.grid_shape(case)
    S, M = int(np.prod(n)), m[0] * m[1]
    planes = n[2] * n[3] * M
    words = (4 + 9 * ((n[0] + 31) // 32) + 3) // 4 * 4
    sizes = [S, S, 64, 12, 64 * len(case["obstacles"]), n[0] * n[1], planes * n[0] * 4,
             planes * ((n[1] + 3) // 4 * 4) * 4, n[2] * m[1] * 4, n[3] * m[0] * 4, 512]
    if fused:
        sizes += [planes * words * 4, planes, n[2] + 1, n[3] + 1]
    return sum(rounded(s) for s in sizes)


def status_under(case, method, budget):
    """Status of creating the problem when its abstraction and `budget` bytes fit."""
    with G.Context(0) as c:
        c.set_memory_budget((64 << 20) - 1)   # below a full-size region of the pool
        a = G.Abstraction(c, case)
        c.set_memory_budget(c.memory_in_use() + budget)
        try:
            G.Problem(c, a, case, method).close()
            status = 0
        except G.GscError as e:
            status = e.status
        a.close()
    return status


@pytest.mark.parametrize("method", [G.METHOD_STORED, G.METHOD_FUSED, G.METHOD_AUTO], ids=["stored", "fused", "auto"])
def test_invalid_candidates_before_memory(method):
    case = C.small_case()
    case.update(candidate="rect", candidate_lb=[-1, -1, -4, 0], candidate_ub=[1, 1, 4, 1],
                obstacles=[[-0.5, -0.5, -4, 0, 0.5, 0.5, 4, 1]])
    need = judged_bytes(case, method != G.METHOD_STORED)
    assert status_under(case, method, need) == 6
    assert status_under(case, method, 64 << 20) == 6
    assert status_under(case, method, need // 2) == 3
    good = C.clone(case, obstacles=[], candidate="ellipse")
    assert status_under(good, method, judged_bytes(good, method != G.METHOD_STORED)) == 3
    assert status_under(good, method, 64 << 20) == 0


def test_unsupported_before_memory():
    """Intervals that the fused method cannot take, asked for by name."""
    case = C.unicycle_grid_case((96, 12, 5, 3), (3, 3))
    case["disturbance_half_width"] = [17.0 * case["state_eta"][0], 0.0, 0.0, 0.0]
    case["constraint"] = "none"
    case["sample_time"] = 1.0
    assert status_under(case, G.METHOD_FUSED, 64 << 20) == 4
    assert status_under(case, G.METHOD_FUSED, judged_bytes(case, True)) == 4
