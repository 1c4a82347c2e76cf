"""The merged table of a linear medium without boundary taper belongs to one step size
and is used only when the last set-up of its slot built it."""
import dataclasses

import numpy as np
import pytest

import scenarios as S
from gpu_helpers import KEYS, solver_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [True, False])
@pytest.mark.parametrize("shape", [(32, 64, 128), (13, 20, 33)])
def test_a_merged_table_of_an_earlier_step_is_not_used(shape, split):
    """Slot 0 without taper at one dz, then with a taper at another, then slot 1 without
    taper: the march is that of a plan whose slot 0 never held the first dz, bit for bit."""
    from angularspectrum_heterogeneous_gb300 import Plan
    kw = dict(S.BASE)
    kw.update(beta=0.0, useSplitStep=split, fluxScheme="kt", useBoundaryLayer=False)
    bare = solver_params(kw)
    taper = dataclasses.replace(bare, useBoundaryLayer=True)
    u0 = S.seeded_field(shape, 5, 1e5).astype(np.float32)
    dz = bare.dZmin
    out = []
    for first in (2.5 * dz, None):
        plan = Plan(shape, bare)
        try:
            if first is not None:
                plan.set_operators(0, first)
            plan.params = taper
            plan.set_operators(0, dz)
            plan.params = bare
            plan.set_operators(1, 0.5 * dz)
            plan.run(u0, 3.0 * dz, dz)
            out.append(plan.outputs())
        finally:
            plan.close()
    for k, a, b in zip(KEYS, *out):
        np.testing.assert_array_equal(a, b, err_msg=k)
