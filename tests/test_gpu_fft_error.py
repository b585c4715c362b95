"""Rounding error of the viscoacoustic K operator: no larger than that of the operator
by direct sums over the prime factors of the lengths, restated here in fp32 (the
transforms, |k| and the scale), for lengths of every kind: prime factors of 17 to
137 (one or several, alone or beside small ones), above 137 (chirp-z), and products
of small primes.

The tolerance is the restated operator's own error on the same fields.
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


def _factors(n):
    out = []
    for p in [4, 2, 3, 5, 7, *range(11, n + 1, 2)]:
        while n % p == 0:
            out.append(p)
            n //= p
    return out


def _direct(re, im, inverse):
    """FFT along axis 0 in fp32, each output of a stage summed from its inputs times the
    roots (real arithmetic: numpy's complex product rounds differently from one
    machine to another)."""
    n = re.shape[0]
    k = np.arange(n)
    tw = np.exp((2j if inverse else -2j) * np.pi * k / n)
    wr, wi = tw.real.astype(np.float32)[:, None], tw.imag.astype(np.float32)[:, None]
    Ns = 1
    for R in _factors(n):
        span = Ns * R
        blk, rem = k // span, k % span
        j = blk * Ns + rem % Ns
        ar, ai = np.zeros_like(re), np.zeros_like(im)
        for r in range(R):
            x, y, e = re[j + r * (n // R)], im[j + r * (n // R)], (r * rem) % span * (n // span)
            ar = ar + (x * wr[e] - y * wi[e])
            ai = ai + (x * wi[e] + y * wr[e])
        re, im, Ns = ar, ai, span
    return re, im


def _direct_k(u, h):
    """K on the pair u[0] + i u[1] (fp32)."""
    f4, (nz, nx) = np.float32, u.shape[1:]
    freq = lambda n: np.fft.fftfreq(n, d=1 / n).astype(f4) * (f4(1) / (f4(n) * f4(h)))
    k = np.sqrt(freq(nz)[:, None] ** 2 + freq(nx)[None] ** 2)
    t = lambda p: (np.ascontiguousarray(p[0].T), np.ascontiguousarray(p[1].T))
    w = _direct(*t(_direct(*t(u), False)), False)
    w = _direct(*t(_direct(k * w[0], k * w[1], True)), True)
    out = np.stack(t(w)) * (f4(1) / (f4(nz) * f4(nx)))
    assert out.dtype == f4
    return out


@pytest.mark.parametrize("nz,nx", [(228, 356), (246, 510), (185, 731), (17, 137), (289, 274), (323, 131), (108, 411),
                                   (278, 389), (500, 1100), (216, 280), (96, 1309)])
def test_error_is_at_most_that_of_direct_sums(dev, nz, nx):
    from seistorch_gb300 import engine
    h = 10.0
    u = np.random.default_rng(nz * 10007 + nx).standard_normal((2, nz, nx)).astype(np.float32)
    kz, kx = np.meshgrid(np.fft.fftfreq(nz, d=h), np.fft.fftfreq(nx, d=h), indexing="ij")
    k = np.sqrt(kz ** 2 + kx ** 2)
    want = np.real(np.fft.ifft2(k * np.fft.fft2(u.astype(np.float64), axes=(-2, -1)), axes=(-2, -1)))
    prop = engine.VacousticPropagator(nz, nx, 0.001, h, 2, 0, False, dev)
    got = prop.kterm(engine.to_pitched(torch.tensor(u, device=dev), prop.pitch).contiguous())[..., :nx].cpu().numpy()
    assert rel_l2(got, want) <= rel_l2(_direct_k(u, h), want)
