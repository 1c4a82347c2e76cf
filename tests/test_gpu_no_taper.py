"""Marches without boundary taper, whose neighbouring spectral stages run as one
(march_step), against the FP64 oracle: Strang and Lie, linear and nonlinear media, with
and without the boundary epilogue and a screen, on fast and any-size planes."""
import numpy as np
import pytest

import oracle.asm_oracle as O
import scenarios as S
import test_gpu_parity as P
from gpu_helpers import KEYS, TOL, oracle_params, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(64, 128, 128), (32, 64, 128), (21, 18, 34), (13, 20, 33)])
@pytest.mark.parametrize("beta", [0.0, 3.5])
@pytest.mark.parametrize("split", [True, False])
@pytest.mark.parametrize("extras", [False, True])
def test_merged_stages(shape, beta, split, extras):
    kw = dict(S.BASE)
    kw.update(beta=beta, useSplitStep=split, fluxScheme="kt", useBoundaryLayer=False,
              propDist=4.5 * kw["dZmin"])
    ex = {}
    if extras:
        kw.update(useFreqWeightedBoundary=True, useSuperAbsorbing=True)
        ex["phaseScreens"] = S._screens(*shape[:2], 5, [1.5 * kw["dZmin"]], [True])
    u0 = S.piston_field(*shape, kw["dX"], kw["dY"], kw["dT"], kw["f0"], 2e6,
                        radius=0.35 * shape[0] * kw["dX"], focus=8e-3)
    res = P._gpu_solve(u0, kw, ex)
    ref = O.solve(u0, oracle_params(kw, ex), "fp64")
    for k, a, r in zip(KEYS, res, ref):
        if k == "zaxis":
            np.testing.assert_array_equal(a, r)
        elif k == "pIloss":  # a difference of two nearly equal sums: relative to the sums
            assert np.linalg.norm(a - r) < 1e-5 * np.linalg.norm(ref[3]), k
        else:
            assert rel(a, r) < TOL[k], (k, rel(a, r))
