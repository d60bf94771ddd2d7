"""Many inputs a slice: more than a block of threads lists at once, and more
columns than it chains (2,048), with one plane a slice and with one an input.
Bit-exact against the oracle."""
import pytest

import gsc_b200 as G
import gsc_cases as C
import oracle as O
from helpers import assert_same_result

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("substeps", [1, 3])
@pytest.mark.parametrize("inputs", [(13, 90), (1, 2048), (1, 2049)])
def test_representatives_of_many_inputs(inputs, substeps):
    case = C.unicycle_grid_case((16, 18, 12, 4), inputs, max_iterations=6)
    case.update(integration_substeps=substeps, sample_time=1.0, input_lb=[-0.4, -3.0], input_ub=[0.4, 3.0],
                input_eta=[0.8 / inputs[0], 6.0 / inputs[1]], disturbance_half_width=[0.0] * 4,
                constraint_params=[1.0, 1.0, 9.0, 1.8], candidate_ellipse=[0.0, -0.6, 1.0, 1.0, 1.5])
    want = O.solve(case)
    assert want["iterations"] > 2
    with G.Context(0) as ctx:
        a = G.Abstraction(ctx, case)
        p = G.Problem(ctx, a, case, G.METHOD_FUSED)
        p.solve()
        got = p.read()
        assert_same_result(got, want, str(inputs))
        assert got["iterations"] == want["iterations"] and got["message"] == want["message"]
