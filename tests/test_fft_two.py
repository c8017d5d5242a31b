"""Transforms on the two-factor lines and the passes built on them, at the lengths where their dispatch and
their tiles change: every radix class (2^a 3^b 5^c up to 16, 25 and 32, and factors 7, 11, 13), equal and
unequal factors, the smallest lines, lengths without two radices (the staged engine), and planes up to the
largest that fits a CTA's shared memory.

The transform bound is 1e-6 in the relative 2-norm: a float32 FFT of n points errs by about
eps log2(n) / 2 = 6e-8 * 9 / 2 per axis; three axes at n = 512 give under 1e-6."""

from __future__ import annotations

import numpy as np
import pytest
from conftest import rel_err

pytestmark = pytest.mark.gpu

G = np.array([0.532, 1.337, 1.2, 0.2], np.float32)
LENGTHS = [4, 6, 10, 14, 22, 26, 34, 62, 66, 78, 90, 96, 126, 154, 160, 182, 200, 208, 250, 286, 300, 320, 336, 352,
           384, 390, 400, 416, 448, 480, 512]


@pytest.mark.parametrize("n", LENGTHS)
def test_transforms_of_every_length_class(cuda, n):
    from qoraholo_b200 import capi

    rng = np.random.default_rng(n)
    x = (rng.standard_normal((3, n, n)) + 1j * rng.standard_normal((3, n, n))).astype(np.complex64)
    for forward, fft in ((True, np.fft.fft2), (False, lambda a: np.fft.ifft2(a) * n * n)):
        d = cuda.from_numpy(x).cuda()
        capi.fft2d(d.data_ptr(), 3, n, forward, 0.5)
        assert rel_err(d.cpu().numpy(), 0.5 * fft(x.astype(np.complex128))) < 1e-6
    nz, ny = 6, 9  # 45 rows: the last tile is ragged
    r = rng.standard_normal((nz - 1, ny, n)).astype(np.float32)
    want = np.fft.rfftn(r.astype(np.float64))
    d, h = cuda.from_numpy(r).cuda(), cuda.empty((nz - 1, ny, n // 2 + 1), dtype=cuda.complex64, device="cuda")
    capi.rfft3(d.data_ptr(), h.data_ptr(), nz - 1, ny, n)
    assert rel_err(h.cpu().numpy(), want) < 1e-6
    back = cuda.empty_like(d)
    h = cuda.from_numpy(want.astype(np.complex64)).cuda()
    capi.irfft3(h.data_ptr(), back.data_ptr(), nz - 1, ny, n, 1.0 / r.size)
    assert rel_err(back.cpu().numpy(), r) < 1e-6


@pytest.mark.parametrize("nx,nz,ny", [(1024, 2, 4), (1024, 2, 7), (1024, 5, 9), (960, 5, 9), (832, 3, 5)])
def test_real_rows_of_the_longest_lines(cuda, nx, nz, ny):
    """Rows whose staged tiles shared memory cuts short (half length 512 = 16 x 32: seven lines, not eight), whole
    and ragged; the bound is the one of the transforms above."""
    from qoraholo_b200 import capi

    r = np.random.default_rng(nx + ny).standard_normal((nz, ny, nx)).astype(np.float32)
    want = np.fft.rfftn(r.astype(np.float64))
    d, h = cuda.from_numpy(r).cuda(), cuda.empty((nz, ny, nx // 2 + 1), dtype=cuda.complex64, device="cuda")
    capi.rfft3(d.data_ptr(), h.data_ptr(), nz, ny, nx)
    assert rel_err(h.cpu().numpy(), want) < 1e-6
    back = cuda.empty_like(d)
    h = cuda.from_numpy(want.astype(np.complex64)).cuda()
    capi.irfft3(h.data_ptr(), back.data_ptr(), nz, ny, nx, 1.0 / r.size)
    assert rel_err(back.cpu().numpy(), r) < 1e-6


def _gp_against_the_oracle(torch, n, nz, amplitude):
    from oracle import qh_oracle as O
    from qoraholo_b200 import capi

    il = O.circular_scan(3, 0.9, G)
    rng = np.random.default_rng(n)
    fields = (rng.standard_normal((3, n, n)) + 1j * rng.standard_normal((3, n, n))).astype(np.complex64)
    fields *= np.float32(amplitude)
    want, _ = O.reconstruct(fields, il, G, nz=nz, iterations=2)
    plan = capi.OdtPlan(n, 3, il, G, nz=nz, iterations=2)
    d, out = torch.from_numpy(fields).cuda(), torch.empty(plan.shape, dtype=torch.float32, device="cuda")
    plan.run(d.data_ptr(), out.data_ptr())
    torch.cuda.synchronize()
    plan.close()
    # 1e-5 of the contrast: ten transforms of 1e-6 each, and two steps that do not amplify them.
    assert rel_err(out.cpu().numpy() - G[1], want - G[1]) < 1e-5


@pytest.mark.parametrize("n", [4, 10, 12, 30, 34, 48, 66, 90, 96, 126, 150, 154, 160, 176, 182, 196, 200, 208, 210, 220,
                               224, 226, 230])
def test_gp_planes_against_the_oracle(cuda, n):
    """GP with whole planes on chip (up to 224: 226 and 230 have no two radices, and 230 would not fit), for
    every class of x factors; four planes, in CTAs of 512 threads."""
    _gp_against_the_oracle(cuda, n, 4, 0.05)


@pytest.mark.parametrize("n,nz", [(10, 150), (66, 150), (90, 160), (96, 160),  # four and more planes per SM: 128 threads
                                  (120, 150), (128, 150), (150, 152), (154, 150), (160, 150),  # two or three: 256
                                  (182, 150), (224, 150)])  # one, in more than one wave: 512
def test_gp_planes_that_fill_the_gpu(cuda, n, nz):
    """More planes than SMs, for each number of planes that an SM holds and so each CTA size. The contrast falls as
    1 / nz and the index is stored in float32, of spacing 1.2e-7 at 1.337: with 0.05, an rms contrast of 2e-4, storing
    it alone is a difference of up to 2.4e-4; with 0.5 nz / 4, an rms contrast of 0.07, of 7e-7."""
    assert nz > cuda.cuda.get_device_properties(0).multi_processor_count
    _gp_against_the_oracle(cuda, n, nz, 0.5 * nz / 4)
