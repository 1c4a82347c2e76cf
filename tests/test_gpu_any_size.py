"""Line transforms and column steps of any length (asg_lines.cuh): every
transform length at the edges of its range, direct and chirp lengths, odd and
even, single-sample tails, against the FP64 oracle."""
import numpy as np
import pytest

import oracle.asm_oracle as O
import scenarios as S
import test_gpu_parity as P
from gpu_helpers import rel

pytestmark = pytest.mark.gpu

# lengths n: the direct four-step sizes, and for each chirp length M = 32 .. 4096 the
# largest n it holds (M / 2) and the smallest (one above the previous M / 2)
LENGTHS = [3, 15, 16, 17, 31, 32, 33, 48, 49, 64, 65, 96, 97, 128, 129, 192, 193, 255, 256, 257,
           288, 289, 384, 385, 512, 513, 576, 768, 769, 1024, 1025, 1536, 2047, 2048]


@pytest.mark.parametrize("nT", LENGTHS)
def test_columns_of_any_length(nT):
    """Every step operator on a 5 x 4 grid (an even column count, whole pairs)."""
    P.test_step_operators(None, (5, 4, nT))


# the same along x and y (lines up to 1024), with an even and an odd nT (with and
# without a Nyquist plane); the other axis and nT leave partial tiles and blocks
@pytest.mark.parametrize("n", [n for n in LENGTHS if n <= 769] + [1000, 1023, 1024])
def test_planes_of_any_size(n):
    P.test_step_operators(None, (n, 5, 9))
    P.test_step_operators(None, (6, n, 8))


@pytest.mark.parametrize("factor", [0.01, 0.2, 0.34, 0.5])
@pytest.mark.parametrize("shape", [(31, 44, 12), (45, 23, 9)])
def test_boundary_bands_of_any_width(shape, factor):
    """The closing epilogue visits the bands only: bands of one sample, bands with a few
    samples between them, bands that meet (same FP32 transforms and tolerance as the step
    operators)."""
    from angularspectrum_heterogeneous_gb300 import Plan
    nX, nY, nT = shape
    kw, u = P._op_case(shape)
    kw["boundaryFactor"] = factor
    p = P.oracle_params(kw)
    plan = Plan(shape, P.solver_params(kw))
    plan.set_operators(0, 1e-4)
    u64 = u.astype(np.float64)
    fw = O.freq_weighted_mask(nX, nY, nT, p.dT, p.f0, factor, "wendland").astype(np.float64)
    wx, wy = (O.boundary_weights(n, O.band_width(n, factor)).astype(np.float64) for n in (nX, nY))
    assert rel(plan.apply_operator(5, u), O.freq_weighted_step(u64, fw)) < 2e-6
    assert rel(plan.apply_operator(6, u), O.super_absorbing_step(
        u64, wx, wy, p.dX, p.dY, p.dT, p.c0, 0.8)) < 2e-6
    plan.close()


@pytest.mark.parametrize("nT", [4, 5, 31, 33, 64, 127, 129, 640, 1000, 1025, 2048])
@pytest.mark.parametrize("flux", ["kt", "ktmm"])
def test_kt_runs_of_any_length(nT, flux):
    """The streamed KT step with runs of every remainder, several columns per block (9)."""
    from angularspectrum_heterogeneous_gb300 import _lib
    N = 3.5 / (2 * 1540.0 ** 3 * 1000.0)
    cols = np.stack([S.seeded_column(nT, s) for s in range(9)]).astype(np.float32)
    kind = _lib.FLUX_KT if flux == "kt" else _lib.FLUX_KT_MINMOD
    out = _lib.flux_columns(cols, kind, N, 4e-4, 1e-8)
    ref = O.flux_kt(cols.astype(np.float64), N, 4e-4, 1e-8, "mc" if flux == "kt" else "minmod")
    assert rel(out, ref) < 2e-6
