"""The gate kernel of the learned step at every column length it takes: 1 to 8 columns per
block with partial blocks, plain sub-cycled columns and coarse steps, against the
FP64 oracle."""
import ctypes as C

import numpy as np
import pytest

import oracle.asm_oracle as O
import scenarios as S
from gpu_helpers import rel

pytestmark = pytest.mark.gpu

N_COEF = 3.5 / (2 * 1540.0 ** 3 * 1000.0)
DZ, DT = 4e-4, 1e-8


def _step(net, cols, flux, target, min_sub):
    import torch
    from angularspectrum_heterogeneous_gb300 import _lib
    a = torch.from_numpy(cols).cuda()
    b = torch.empty_like(a)
    n = C.c_int(-1)
    _lib.check(_lib.load().asg_flux_columns_learned(
        net.h, C.c_void_p(a.data_ptr()), C.c_void_p(b.data_ptr()), cols.shape[0], cols.shape[1],
        flux, N_COEF, DZ, DT, target, 1024, min_sub, 10.0, C.byref(n),
        C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return b.cpu().numpy(), n.value


@pytest.mark.parametrize("nT", range(128, 1025, 128))
@pytest.mark.parametrize("ncols", [1, 9, 611, 2451])
def test_gate_columns(nT, ncols):
    """FP32 KT steps: the tolerance of the column tests (2e-6 for one step), growing with the
    square root of the sub-steps' roundings."""
    from angularspectrum_heterogeneous_gb300 import _lib
    from angularspectrum_heterogeneous_gb300 import corrector as CR
    cols = np.stack([S.seeded_column(nT, s) for s in range(min(ncols, 13))]).astype(np.float32)
    cols = cols[np.arange(ncols) % len(cols)]
    net = CR.Corrector(np.zeros_like(CR.init_params(1)))  # no correction: the coarse step alone
    try:
        for flux, lim in ((_lib.FLUX_KT, "mc"), (_lib.FLUX_KT_MINMOD, "minmod")):
            c64 = cols[:13].astype(np.float64)
            coarse = O.flux_kt(c64, N_COEF, DZ, DT, lim)
            out, n = _step(net, cols, flux, 1e-3, 1)
            cfl = N_COEF / DT * np.abs(cols).max(axis=1) * DZ
            assert n == ncols and cfl.max() <= 0.5
            for k in range(min(ncols, 13)):
                assert rel(out[k], coarse[k]) < 2e-6, k
            target = float(cfl.max()) / 2.5  # up to three sub-steps
            out, n = _step(net, cols, flux, target, 10 ** 6)
            assert n == 0
            for k in range(min(ncols, 13)):
                sub = int(np.ceil(np.float32(cfl[k]) / np.float32(target)))
                r = c64[k:k + 1]
                for _ in range(max(sub, 1)):
                    r = O.flux_kt(r, N_COEF, DZ / max(sub, 1), DT, lim)
                assert rel(out[k], r[0]) < 2e-6 * np.sqrt(max(sub, 1)), k
            # every copy of a column takes the same path
            for i in range(len(c64), ncols):
                assert np.array_equal(out[i], out[i % len(c64)]), i
    finally:
        net.close()
