"""A rejected plan leaves no CUDA error behind: the next plan works."""
import numpy as np
import pytest

import scenarios as S
from gpu_helpers import solver_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [(64, 1, 64), (9, 2000, 9), (9, 9, 3001), (1100, 300, 9)])
def test_next_plan_works(bad):
    from angularspectrum_heterogeneous_gb300 import Plan
    from angularspectrum_heterogeneous_gb300._lib import ASGError
    kw = dict(S.BASE)
    good = (12, 10, 31)
    u0 = S.seeded_field(good, 2, 1e5).astype(np.float32)
    with pytest.raises(ASGError) as e:
        Plan(bad, solver_params(kw))
    assert e.value.code == -2  # ASG_ERR_SHAPE
    plan = Plan(good, solver_params(kw))
    try:
        plan.set_operators(0, kw["dZmin"])
        plan.run(u0, 2 * kw["dZmin"], kw["dZmin"])
        assert np.isfinite(plan.outputs()[0]).all()
    finally:
        plan.close()
