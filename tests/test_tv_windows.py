"""The two-step FGP form in windows and tall tiles (bitwise the stored-r form and the oracle): short rows of every
tile height, rows just over one tile, several windows with a short last one, ragged last tiles in y, fewer
planes than the march runs ahead, odd and even step counts."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _prox(torch, capi, b, p, lam, inner, form):
    d = torch.from_numpy(b).cuda()
    work = torch.zeros((12, *b.shape), device="cuda")
    work[:3] = torch.from_numpy(p).cuda()
    x = torch.empty_like(d)
    try:
        capi.tv_form(form)
        capi.tv_prox_workspace(d.data_ptr(), x.data_ptr(), work.data_ptr(), 12, *b.shape, lam, inner)
        torch.cuda.synchronize()
    finally:
        capi.tv_form(0)
    return x.cpu().numpy(), work[:3].cpu().numpy()


@pytest.mark.parametrize("shape,inner", [((5, 7, 8), 4), ((1, 40, 96), 2), ((9, 33, 128), 5), ((3, 29, 132), 4),
                                         ((6, 40, 160), 4), ((7, 23, 180), 3), ((4, 30, 192), 4), ((2, 17, 208), 2),
                                         ((6, 20, 256), 4), ((6, 20, 260), 5), ((5, 19, 320), 4), ((4, 17, 384), 2),
                                         ((5, 9, 516), 4), ((3, 12, 1024), 2)])
def test_windows_are_bitwise_the_one_step_form(cuda, shape, inner):
    from oracle import qh_oracle as O
    from qoraholo_b200 import capi

    rng = np.random.default_rng(sum(shape))
    b = (3.0 * rng.random(shape)).astype(np.float32)
    p = (rng.uniform(-0.5, 0.5, (3, *shape))).astype(np.float32)
    one = _prox(cuda, capi, b, p, 0.7, inner, 1)
    for form in (0, 3):
        two = _prox(cuda, capi, b, p, 0.7, inner, form)
        assert np.array_equal(one[0], two[0]) and np.array_equal(one[1], two[1]), form
    dual = [c.copy() for c in p]
    want = O.tv_prox(b, dual, 0.7, inner)
    assert np.array_equal(two[0], want) and all(np.array_equal(two[1][i], dual[i]) for i in range(3))
