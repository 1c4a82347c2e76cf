"""Small planes, one block each: every pass radix along x and y, narrow planes of long axes up to
beyond 1024 rows, the largest plane of the rule and the first beyond, with and without a
Nyquist plane, against the FP64 oracle (step operators and their tolerance)."""
import numpy as np
import pytest

import oracle.asm_oracle as O
import scenarios as S
import test_gpu_parity as P
from gpu_helpers import KEYS, TOL, oracle_params, rel

pytestmark = pytest.mark.gpu

SIZES = list(range(2, 19)) + [20, 21, 22, 24, 25, 26, 27, 28, 30, 32, 33, 34, 35, 36, 39, 42, 44,
                              45, 48, 49, 51, 52]


@pytest.mark.parametrize("n", SIZES)
def test_square_planes(n):
    P.test_step_operators(None, (n, n, 8))


@pytest.mark.parametrize("shape", [(4, 1024, 9), (1024, 4, 8), (2, 729, 8), (625, 3, 9), (8, 400, 8),
                                   (512, 8, 9), (1536, 3, 8), (7, 680, 8), (17, 19, 9), (19, 8, 8),
                                   (5, 48, 7), (75, 16, 8), (12, 121, 9), (20, 100, 8),
                                   (3, 1000, 9), (1000, 3, 8),
                                   # sums of odd primes spread over the block: partly and
                                   # wholly filled, beside another pass, one line too many
                                   (37, 3, 8), (3, 41, 9), (61, 8, 8), (8, 53, 9), (16, 23, 8),
                                   (31, 16, 9), (17, 31, 8), (46, 5, 9), (4, 58, 8), (19, 19, 9),
                                   (23, 11, 8), (38, 6, 9), (2, 43, 8), (67, 3, 8), (4, 79, 9),
                                   # line passes with fewer than eight columns
                                   (381, 2, 8), (331, 3, 9), (997, 4, 8), (83, 5, 9)])
def test_narrow_planes(shape):
    P.test_step_operators(None, shape)


@pytest.mark.parametrize("shape", [(16, 16, 256), (21, 20, 33), (2, 130, 64)])
@pytest.mark.parametrize("obl", [False, True])
def test_small_solves(shape, obl):
    """Whole marches with screens, boundary extras and beam obliquity."""
    kw = dict(S.BASE)
    kw.update(fluxScheme="kt", useFreqWeightedBoundary=True, useSuperAbsorbing=True,
              useNonlinearityObliquity=obl, propDist=6.5 * kw["dZmin"])
    ex = {"phaseScreens": S._screens(*shape[:2], 5, [1.5 * kw["dZmin"]], [True])}
    u0 = S.seeded_field(shape, 4, 1e6).astype(np.float32)
    res = P._gpu_solve(u0, kw, ex)
    ref = O.solve(u0, oracle_params(kw, ex), "fp64")
    for k, a, r in zip(KEYS, res, ref):
        if k == "zaxis":
            np.testing.assert_array_equal(a, r)
        elif k == "pIloss":  # a difference of two sums (after: pI), relative to the first
            assert np.linalg.norm(a - r) < 1e-5 * np.linalg.norm(ref[3] + ref[4]), k
        else:
            assert rel(a, r) < TOL[k], (k, rel(a, r))
