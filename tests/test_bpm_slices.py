"""The BPM slice passes at the sides where their dispatch changes (staged below 48 and without two radices,
the register engine at 64, 128 and 256, the two-factor lines elsewhere, in each radix class) and with view
counts around a group of the row passes, against the oracle."""

from __future__ import annotations

import numpy as np
import pytest
from conftest import rel_err

pytestmark = pytest.mark.gpu

G = np.array([0.532, 1.337, 1.2, 0.2], np.float32)


@pytest.mark.parametrize("n,count", [(46, 3), (48, 1), (62, 3), (64, 33), (66, 17), (78, 3), (100, 16), (154, 2),
                                     (160, 17), (200, 2), (240, 3)])
def test_slice_passes_match_the_oracle(cuda, n, count):
    from oracle import qh_oracle as O
    from qoraholo_b200.autograd import BpmModel

    rng = np.random.default_rng(n)
    nz = 5
    il = O.circular_scan(count, 0.9, G)
    ri = (G[1] + 0.03 * rng.random((nz, n, n))).astype(np.float32)
    r = (rng.standard_normal((count, n, n)) + 1j * rng.standard_normal((count, n, n))).astype(np.complex64) * 0.1
    want = O.bpm_forward(ri, il, G)
    want_grad = O.bpm_vjp((ri - G[1]).astype(np.float32), r, O.bpm_tables(n, nz, il, G))
    grads = []
    for every in (2, 5):  # bitwise the same gradient whatever is stored
        x = cuda.from_numpy(ri).cuda().requires_grad_(True)
        y = BpmModel(nz, n, il, G, checkpoint_every=every)(x)
        y.backward(cuda.from_numpy(r).cuda())
        grads.append(x.grad.cpu().numpy())
    # 2 transforms per slice of 1e-6 at most, forward; as many again back.
    assert rel_err(y.detach().cpu().numpy(), want) < 1e-5
    assert rel_err(grads[0], want_grad) < 2e-5
    assert np.array_equal(grads[0], grads[1])


def test_passes_over_the_views_agree_with_one_pass(cuda):
    """As many views as the plan takes in two passes: fields bitwise those of one pass, the gradient
    up to the order in which the passes' sums are added (two passes of float32 sums: 4e-7)."""
    from oracle import qh_oracle as O
    from qoraholo_b200.autograd import BpmModel

    n, nz, count = 256, 3, 49  # 86 MB of state
    rng = np.random.default_rng(3)
    il = O.circular_scan(count, 0.9, G)
    ri = cuda.from_numpy((G[1] + 0.03 * rng.random((nz, n, n))).astype(np.float32)).cuda()
    out = []
    for chunk in (0, count):
        x = ri.clone().requires_grad_(True)
        y = BpmModel(nz, n, il, G, checkpoint_every=2, chunk=chunk)(x)
        y.backward(y.detach() - 1)
        out.append((y.detach().cpu().numpy(), x.grad.cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0])
    assert rel_err(out[0][1], out[1][1]) < 4e-7


@pytest.mark.parametrize("n,count,passes", [(256, 49, 2), (256, 52, 2), (384, 20, 2),  # 72 to 112 MB of state
                                            (256, 40, 1), (260, 36, 1),  # halves would make another group of views
                                            (352, 20, 1), (512, 18, 1), (512, 30, 1),  # below, above, several passes
                                            (160, 96, 1), (240, 49, 1), (272, 33, 1)])  # small sides, no two radices
def test_the_default_splits_the_views_only_where_it_pays(cuda, n, count, passes):
    """By the buffers the plan holds: those of a plan told how many views a pass takes."""
    from oracle import qh_oracle as O
    from qoraholo_b200.autograd import BpmPlan

    il = O.circular_scan(count, 0.9, G)
    plans = [BpmPlan(2, n, il, G, chunk=c, checkpoint_every=1) for c in (0, -(-count // passes), count)]
    held = [p.device_bytes for p in plans]
    assert held[0] == held[1] and (held[0] == held[2]) == (passes == 1)
