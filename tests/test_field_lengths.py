"""Field extraction at hologram and output sides of every engine (two-factor lines in each radix class, 1024 = 32 x
32 columns, staged lengths with large primes), with the window at the edge of the spectrum, and the complex
Ewald mapping at axial sides around its tiles."""

from __future__ import annotations

import numpy as np
import pytest
from conftest import rel_err

pytestmark = pytest.mark.gpu

G = np.array([0.532, 1.337, 1.2, 0.2], np.float32)


@pytest.mark.parametrize("n,m", [(16, 8), (34, 16), (60, 62), (64, 64), (100, 48), (126, 90), (128, 128), (154, 78),
                                 (200, 96), (302, 150), (400, 200), (512, 256), (1024, 384)])
def test_fields_match_the_oracle(cuda, n, m):
    import qoraholo_b200 as qh
    from oracle import qh_oracle as O

    m = min(m, n)
    h = np.random.default_rng(n).random((2, n, n)).astype(np.float32)
    for center in ((n // 4 + 1, n // 4), (3, n // 2 - 2), (-2, -n // 4)):  # inside, across the edge, negative kx
        kw = dict(center=tuple(map(float, center)), radius=m / 2 - 1.0, output_size=m)
        # Three transforms of about 3e-7 each on noise whose window holds a fair share of the energy.
        assert rel_err(qh.extract_fields(h, **kw), O.extract_fields(h, **kw)) < 2e-6


@pytest.mark.parametrize("n,nz,count", [(6, 2, 1), (10, 8, 33), (16, 64, 70), (8, 512, 5), (8, 514, 5), (6, 1024, 3),
                                        (6, 1030, 3)])
def test_complex_mapping_is_bit_identical(cuda, n, nz, count):
    from oracle import qh_oracle as O
    from qoraholo_b200 import capi

    rng = np.random.default_rng(n + nz)
    il = O.circular_scan(count, 0.9, G) if count > 1 else np.zeros((1, 2), np.float32)
    sp = (rng.standard_normal((count, n, n)) + 1j * rng.standard_normal((count, n, n))).astype(np.complex64)
    pre, pim, w = O.ewald_map(sp, il, O.make_grid(n, nz, G))
    hit = w > 0
    want = (np.where(hit, pre / np.where(hit, w, 1), pre) + 1j * np.where(hit, pim / np.where(hit, w, 1), pim))
    d = cuda.from_numpy(sp).cuda()
    pot = cuda.empty((nz, n, n), dtype=cuda.complex64, device="cuda")
    mask = cuda.empty((nz, n, n), dtype=cuda.uint8, device="cuda")
    filled = cuda.zeros(1, dtype=cuda.int64, device="cuda")
    capi.ewald_map(d.data_ptr(), count, n, nz, il, G, False, pot.data_ptr(), mask.data_ptr(), filled.data_ptr())
    assert np.array_equal(pot.cpu().numpy(), want.astype(np.complex64))
    assert np.array_equal(mask.cpu().numpy().astype(bool), hit) and int(filled) == int(hit.sum())
