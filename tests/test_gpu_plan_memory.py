"""Device memory of a plan on the L2-exchange planes: its exchange scratch holds the CTA groups
that can run at once, whatever the tuning knobs say."""
import numpy as np
import pytest

import scenarios as S
from gpu_helpers import solver_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(128, 128, 128), (192, 192, 128), (256, 256, 128)])
def test_exchange_scratch_holds_the_resident_groups(shape):
    import torch
    from angularspectrum_heterogeneous_gb300 import Plan
    nX, nY, nT = shape
    kw = dict(S.BASE)
    Plan(shape, solver_params(kw)).close()  # kernels and constant tables are loaded
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    plan = Plan(shape, solver_params(kw))
    try:
        used = before - torch.cuda.mem_get_info()[0]
        planes = nT // 2 + 1
        field, spec = 4 * nX * nY * nT, 8 * nX * nY * planes
        table = 8 * ((nX + 1) // 2) * ((nY + 1) // 2) * planes
        # 16 rows and 256 threads per CTA: at most 8 CTAs per SM, X / 32 CTAs and two
        # half-planes of 8 bytes per sample per group; 2 MB granules for some forty buffers
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        groups = min(2 * planes, 8 * sms // (nX // 32))
        scratch = min(groups * 8 * nX * nY, 40 << 20)
        assert used < field + spec + table + scratch + (16 << 20), used / 2**20
    finally:
        plan.close()


@pytest.mark.parametrize("shape", [(64, 128, 192), (192, 192, 128), (256, 256, 128)])
def test_any_group_cap_gives_the_same_march(shape):
    """Caps below and above the resident groups, clusters and cooperative launches: bit-identical."""
    from angularspectrum_heterogeneous_gb300 import Plan
    kw = dict(S.BASE)
    kw.update(fluxScheme="kt", useFreqWeightedBoundary=True, useSuperAbsorbing=True)
    u0 = S.seeded_field(shape, 7, 1e6).astype(np.float32)
    plan = Plan(shape, solver_params(kw))
    try:
        plan.set_operators(0, kw["dZmin"])
        out = []
        for sync in (1, 2, 3):
            for cap in (0, 1, 63, 64):
                plan.set_tuning(dict(t_cols_flux=0, t_cols_plain=0, t_cols_stats=0,
                                     xy_clusters=cap, xy_clusters_closing=cap, xy_sync=sync))
                plan.run(u0, 2 * kw["dZmin"], kw["dZmin"])
                out.append(plan.outputs())
        for o in out[1:]:
            for a, b in zip(out[0], o):
                np.testing.assert_array_equal(a, b)
    finally:
        plan.close()
