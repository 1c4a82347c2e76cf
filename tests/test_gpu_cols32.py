"""Column passes with 32 columns per block: bit-identical to 16 in every mode (flux,
taper, statistics, first and last step), at the smallest and ragged grids they take."""
import numpy as np
import pytest

import scenarios as S
from gpu_helpers import solver_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 16, 128), (6, 48, 192), (32, 64, 256), (64, 128, 256)])
@pytest.mark.parametrize("flux", ["kt", "rusanov"])
def test_32_columns_per_block(shape, flux):
    from angularspectrum_heterogeneous_gb300 import Plan
    kw = dict(S.BASE)
    kw.update(fluxScheme=flux, propDist=3 * kw["dZmin"])
    u0 = S.seeded_field(shape, 3, 2e6).astype(np.float32)
    plan = Plan(shape, solver_params(kw))
    out = {}
    try:
        plan.set_operators(0, kw["dZmin"])
        for cols in (16, 32):
            plan.set_tuning(dict(t_cols_flux=cols, t_cols_plain=cols, t_cols_stats=cols,
                                 xy_clusters=0, xy_clusters_closing=0, xy_sync=0, t_prefetch=2))
            plan.run(u0, kw["propDist"], kw["dZmin"])
            out[cols] = plan.outputs()
    finally:
        plan.close()
    for a, b in zip(out[16], out[32]):
        np.testing.assert_array_equal(a, b)
