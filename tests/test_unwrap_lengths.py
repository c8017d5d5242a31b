"""The unwrap at side lengths of every engine: two-factor lines in each radix class, lines whose second factor
is a direct sum (prime factors of 17 and more, even and odd lengths, a prime half length), the register and the
staged engine beside them, the smallest sides; single, batched and without allocation."""

from __future__ import annotations

import numpy as np
import pytest
from conftest import rel_err
from test_batch import phase_map

pytestmark = pytest.mark.gpu

SHAPES = [(2, 8), (8, 10), (6, 34), (34, 38), (62, 74), (66, 70), (96, 200), (120, 160), (126, 128), (158, 346),
          (202, 106), (136, 248), (290, 272), (322, 578), (512, 610), (632, 640), (646, 104), (1018, 130)]


@pytest.mark.parametrize("ny,nx", SHAPES)
def test_every_engine_matches_the_oracle(cuda, ny, nx):
    from oracle import qh_oracle as O
    from qoraholo_b200 import capi

    img = phase_map(np.random.default_rng(ny * nx), ny, nx)
    want = O.unwrap(img[None])[0]
    d, out = cuda.from_numpy(img).cuda(), cuda.empty((ny, nx), device="cuda")
    capi.unwrap_noalloc(d.data_ptr(), out.data_ptr(), 1, ny, nx)
    # The eigenvalues are the oracle's floats, so only the transforms' rounding differs; it shows in the lowest
    # modes, whose eigenvalues are smallest: 1.3e-6 at most with the images transposed.
    assert rel_err(out.cpu().numpy(), want) < 1e-5


def test_batched_single_and_no_allocation_are_bitwise_the_same(cuda):
    import qoraholo_b200 as qh
    from qoraholo_b200 import capi

    rng = np.random.default_rng(7)
    images = [phase_map(rng, ny, nx) for ny, nx in SHAPES]
    plan = capi.UnwrapBatch(SHAPES)
    d = cuda.from_numpy(plan.pack(images)).cuda()
    out, alone = cuda.empty_like(d), cuda.empty_like(d)
    plan.run(d.data_ptr(), out.data_ptr())
    for off, (ny, nx) in zip(plan.offsets, SHAPES):
        capi.unwrap_noalloc(d.data_ptr() + 4 * off, alone.data_ptr() + 4 * off, 1, ny, nx)
    cuda.cuda.synchronize()
    plan.close()
    assert cuda.equal(out, alone)
    for img, got in zip(images, plan.unpack(out.cpu().numpy())):
        assert np.array_equal(got, qh.unwrap(img)), img.shape
