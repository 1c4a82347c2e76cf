"""KT steps on short columns, whose sub-steps stay in registers: every number of samples per
lane, full and ragged last lanes, one length beyond, sub-cycled per column, against the
FP64 oracle."""
import numpy as np
import pytest

import oracle.asm_oracle as O
import scenarios as S
from gpu_helpers import rel

pytestmark = pytest.mark.gpu

LENGTHS = [3, 4, 31] + [n for k in range(1, 9) for n in (32 * k, 32 * k + 1)] + \
    [50, 90, 120, 150, 180, 210, 250]


@pytest.mark.parametrize("nT", LENGTHS)
@pytest.mark.parametrize("flux", ["kt", "ktmm"])
def test_sub_cycled_short_columns(nT, flux):
    """One column each of 1, 2, .. 9 sub-steps (11 columns: a partial block).  Tolerance: the 2e-6
    of one step (test_kt_runs_of_any_length) per root of the number of steps."""
    from angularspectrum_heterogeneous_gb300 import _lib
    N, dz, dt = 3.5 / (2 * 1540.0 ** 3 * 1000.0), 4e-4, 1e-8
    cols = np.stack([S.seeded_column(nT, s) for s in range(11)])
    steps = [1, 2, 3, 4, 5, 6, 7, 8, 9, 1, 2]
    target = 0.02
    for c, k in zip(cols, steps):  # CFL numbers in the middle of each count
        c *= (k - 0.5) * target / (N / dt * dz * np.abs(c).max())
    cols = cols.astype(np.float32)
    kind = _lib.FLUX_KT if flux == "kt" else _lib.FLUX_KT_MINMOD
    out = _lib.flux_columns(cols, kind, N, dz, dt, cfl_target=target)
    for i, k in enumerate(steps):
        r = cols[i:i + 1].astype(np.float64)
        for _ in range(k):
            r = O.flux_kt(r, N, dz / k, dt, "mc" if flux == "kt" else "minmod")
        assert rel(out[i], r[0]) < 2e-6 * np.sqrt(k), (i, k)
