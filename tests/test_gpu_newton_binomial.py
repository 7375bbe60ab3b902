"""The Newton step of x^3 + c0 and the early answers of settled states, against the oracle, at iteration limits around
the tests (steps 10, 10 + limit / 10, ...) and with polynomials on both sides of the rule (c0 = 0, a linear term, c3 not
1, a c0 that is no binary32 number); frames through the origin and the axes, where f' vanishes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests.gpu_util import pitched, read_pixels, same_pixels  # noqa: E402
from tests.test_gpu_reference_mode import rect_for  # noqa: E402

ROOTS = [1, 0, -0.5, 0.86602540378, -0.5, -0.86602540378]


@pytest.mark.parametrize("max_iter", [1, 9, 10, 11, 30, 31, 57, 200])
@pytest.mark.parametrize("coeffs", [[-1, 0, 0, 1], [-0.1, 0, 0, 1], [0, 0, 0, 1], [-1, 0, 0, 2], [2, -2, 0, 1]])
@pytest.mark.parametrize("kind", [2, 3, 4])
def test_binomial_matches_oracle(cuda, oracle, kind, coeffs, max_iter):
    import chaos_gb300 as cg
    w, h = 41, 33
    rect = rect_for((0.0, 0.0), 4.0, w, h)
    m = cg.Module({2: "newton_wired", 3: "newton_generic", 4: "newton_iterations"}[kind])
    if kind != 2:
        m.write_constant("coefficients", np.array(coeffs, dtype=np.float64).tobytes())
        m.write_constant("roots", np.array(ROOTS, dtype=np.float64).tobytes())
    oracle.set_newton(ROOTS, coeffs, 11)
    for dbl in (False, True):
        buf, pitch = pitched(cuda, w, h)
        m.render_main(buf.data_ptr(), pitch, w, h, rect, max_iter, 2.0, 1, double=dbl)
        want = oracle.render_main(kind, dbl, 1, w, h, rect, max_iter, 2.0, 1)
        assert not same_pixels(read_pixels(buf, w), want).any(), dbl
    oracle.set_newton()
