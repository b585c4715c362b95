"""The viscoacoustic K operator (sgb_vacoustic_kterm) over the lengths its
transforms treat differently: products of the register radices (2, 3, 4, 5, 7,
8, 10, 11, 13), lengths of one pass or none, chirp-z lengths (a prime factor
above 13) from the smallest to the largest, and lengths whose chirp-z does not
fit in shared memory; odd shot counts, rows that do not fill a CTA.

Tolerance against numpy's float64 FFT: an fp32 transform of length n is off by
about eps sqrt(log2 n) per pass pair; the chirp-z pads to M < 3n and does four.
Eight such transforms of at most 2^15 points stay below 8 x 4 x 6e-8 = 2e-6 of
the norm.
"""
import numpy as np
import pytest
import torch

from tests.golden_cases import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from seistorch_gb300 import _native
    _native.load(build_if_missing=False)
    return torch.device("cuda:0")


@pytest.mark.parametrize("shape", [(3, 500, 1100), (2, 169, 1001), (1, 64, 1024), (5, 24, 6), (1, 1, 7), (1, 13, 1),
                                   (2, 17, 356), (1, 251, 401), (1, 2, 4099), (2, 4099, 9), (1, 6911, 3), (1, 3, 7001),
                                   (1, 7001, 5), (1, 8192, 4), (1, 4, 8192)])
def test_k_operator_lengths(dev, shape):
    from seistorch_gb300 import engine
    B, nz, nx = shape
    h = 10.0
    rng = np.random.default_rng(nz * 10007 + nx)
    u1, u2 = rng.standard_normal((2, B, nz, nx))
    post = rng.standard_normal((nz, nx))
    kz, kx = np.meshgrid(np.fft.fftfreq(nz, d=h), np.fft.fftfreq(nx, d=h), indexing="ij")
    k = np.sqrt(kz ** 2 + kx ** 2)
    want = post * np.real(np.fft.ifft2(k * np.fft.fft2(u1 - u2, axes=(-2, -1)), axes=(-2, -1)))
    prop = engine.VacousticPropagator(nz, nx, 0.001, h, 2, 0, False, dev)
    pit = lambda a: engine.to_pitched(torch.tensor(a, dtype=torch.float32, device=dev), prop.pitch).contiguous()
    got = prop.kterm(pit(u1), pit(u2), post=pit(post))
    assert torch.all(got[..., nx:] == 0)
    assert rel_l2(got[..., :nx].cpu().numpy(), want) < 2e-6
