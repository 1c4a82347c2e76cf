"""Every compiled line transform at the edges of its lengths, along t, x and y, against the
FP64 oracle.  The lengths come from the library's own choice (line_plans.py)."""
import pytest

import line_plans as L
import test_gpu_parity as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nT", L.edge_lengths())
def test_columns(nT):
    """Tolerance of the step operators, on a 5 x 4 grid (whole pairs of columns)."""
    P.test_step_operators(None, (5, 4, nT))


# the other axis and nT leave partial tiles and blocks; nT with and without a Nyquist plane
@pytest.mark.parametrize("n", [n for n in L.edge_lengths() if n <= 1024])
def test_planes(n):
    P.test_step_operators(None, (n, 37, 9))
    P.test_step_operators(None, (38, n, 8))
