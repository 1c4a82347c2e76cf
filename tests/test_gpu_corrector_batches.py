"""Gradients of large training batches, where every persistent loop of the training kernels
takes several rounds: the columns are independent, so a batch's loss and gradients are the
means of its parts', each small enough for one round (and those match the oracle)."""
import numpy as np
import pytest

import oracle.corrector as OC
from test_gpu_corrector import _batch, _oracle_params, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nT,ncols,part", [(512, 1024, 8), (128, 3328, 26), (1024, 416, 13)])
def test_a_batch_is_the_mean_of_its_parts(nT, ncols, part):
    """The parts number a power of two, so their scaled gradients are rounded to BF16 alike and only
    FP32 sums over positions differ: each side adds at most a few thousand terms in a row, an
    error of 2^-24 sqrt(4096) = 4e-6 of the terms' size; 1e-5 of the mean size of the parts'
    gradients covers both."""
    import torch
    from angularspectrum_heterogeneous_gb300 import corrector as CR
    net = CR.Corrector(CR.init_params(11, last_scale=1.0))
    try:
        x, tg, mk = _batch(ncols, nT, 5)
        mk[:, nT // 2 - 3:nT // 2] = 0.0
        d = [torch.from_numpy(a).cuda() for a in (x, tg, mk)]
        loss, g = net.train_step(*d, lr=0.0, want_grad=True)
        parts = ncols // part
        assert parts * part == ncols and parts & (parts - 1) == 0
        ls, gs, size = 0.0, 0.0, {}
        for k in range(parts):
            a, b = k * part, (k + 1) * part
            l, h = net.train_step(*[t[a:b].contiguous() for t in d], lr=0.0, want_grad=True)
            ls, gs = ls + l / parts, gs + h.astype(np.float64) / parts
            for name, v in CR.to_dict(h).items():
                size[name] = size.get(name, 0.0) + np.linalg.norm(v) / parts
        assert abs(loss - ls) < 1e-6 * ls
        m = CR.to_dict(gs)
        for name, v in CR.to_dict(g).items():
            assert np.linalg.norm(v - m[name]) < 1e-5 * size[name], name
    finally:
        net.close()


@pytest.mark.parametrize("nT,ncols", [(128, 8), (512, 24), (1024, 3)])
def test_parts_match_the_oracle(nT, ncols):
    """Tolerances of test_gradients_match_oracle (BF16 activations and weights)."""
    import torch
    from angularspectrum_heterogeneous_gb300 import corrector as CR
    theta = CR.init_params(11, last_scale=1.0)
    net = CR.Corrector(theta)
    try:
        x, tg, mk = _batch(ncols, nT, 6)
        loss, g = net.train_step(*[torch.from_numpy(a).cuda() for a in (x, tg, mk)], lr=0.0,
                                 want_grad=True)
        lr_, gr = OC.loss_and_grads(x, tg, mk, _oracle_params(theta, True))
        assert abs(loss - lr_) / lr_ < 2e-2
        gd = CR.to_dict(g)
        for name, _ in CR.SHAPES:
            a, b = gd[name].ravel(), gr[name].ravel()
            cos = float(a @ b / (np.linalg.norm(a) * np.linalg.norm(b) + 1e-30))
            assert cos > 0.995 and _rel(a, b) < 8e-2, (name, cos, _rel(a, b))
    finally:
        net.close()
