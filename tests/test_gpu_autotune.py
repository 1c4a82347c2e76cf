"""The autotuner compares times of passes that the march launches: a knob whose pass a
linear march without taper leaves out keeps its default."""
import numpy as np
import pytest

import scenarios as S
from gpu_helpers import solver_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extras", [False, True])
def test_knobs_of_passes_left_out_keep_their_default(extras):
    from angularspectrum_heterogeneous_gb300 import Plan, solver
    shape = (64, 128, 128)  # L2 planes; 32 columns per block by default
    kw = dict(S.BASE)
    kw.update(beta=0.0, useSplitStep=True, fluxScheme="kt", useBoundaryLayer=False,
              useFreqWeightedBoundary=extras, useSuperAbsorbing=extras)
    u0 = S.seeded_field(shape, 9, 1e5).astype(np.float32)
    plan = Plan(shape, solver_params(kw))
    try:
        plan.set_operators(0, kw["dZmin"])
        plan.set_tuning(dict(t_cols_flux=0, t_cols_plain=0, t_cols_stats=0, xy_clusters=0))
        default = plan.get_tuning()
        plan.run(u0, 2 * kw["dZmin"], kw["dZmin"])
        ref = plan.outputs()
        launches = {k: v[1] for k, v in plan.kernel_stats().items()}
        assert launches["t_nonlin"] == launches["t_mid"] == 0
        # the boundary epilogue of L2 planes keeps the diffraction in a pass of its own
        assert (launches["xy_A"] > 0) == extras and launches["xy_C"] > 0
        chosen = plan.autotune(u0, kw["dZmin"], steps=2)
        assert default["t_cols_flux"] != 8
        for k in ("t_cols_flux", "t_cols_plain"):
            assert chosen[k] == default[k], k
        plan.run(u0, 2 * kw["dZmin"], kw["dZmin"])
        for a, b in zip(ref, plan.outputs()):
            np.testing.assert_array_equal(a, b)
    finally:
        plan.close()
        solver.TUNING_CACHE.clear()
