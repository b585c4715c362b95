"""Infinities and NaN in the weight gradients of the input and output convolutions:
a pixel beyond the image takes no part, nor (input convolution) one whose gradient is
0, so every sum is the one that PyTorch forms over the remaining products, non-finite
ones included.

The finite sums of the 455 products at most are compared to 1e-5 of the largest.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def N():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from seistorch_gb300 import _native
    _native.load(build_if_missing=False)
    return _native


def _sums(v, s, sign, skip_zero):
    """dW[c][k] = sum_p v[p][c] s[p + d_k] over the pixels that take part, float64."""
    h, w, c = v.shape
    out = torch.zeros(c, 9, dtype=torch.float64, device=v.device)
    vd, sd = v.double(), s.double()
    for k in range(9):
        dy, dx = sign * (k // 3 - 1), sign * (k % 3 - 1)
        y0, y1, x0, x1 = max(0, -dy), min(h, h - dy), max(0, -dx), min(w, w - dx)
        a, b = vd[y0:y1, x0:x1], sd[y0 + dy:y1 + dy, x0 + dx:x1 + dx, None]
        p = a * b
        if skip_zero:
            p = torch.where(a == 0, torch.zeros_like(p), p)
        out[:, k] = p.sum((0, 1))
    return out


def _same(got, want):
    got = got.double()
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.isinf(got), torch.isinf(want)) and torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
    f = torch.isfinite(want)
    assert not f.any() or (got[f] - want[f]).abs().max() < 1e-5 * want[f].abs().max()


INF, NAN = float("inf"), float("nan")
# (value in the image, its pixel, value in the NHWC tensor, its pixel)
CASES = [(INF, (3, 30), None, None), (-INF, (0, 0), None, None), (NAN, (6, 64), None, None), (None, None, INF, (0, 64)),
         (None, None, -INF, (6, 0)), (None, None, NAN, (3, 20)), (INF, (6, 63), INF, (0, 5)), (None, None, None, None)]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("c,cstride", [(32, 32), (5, 11)])
def test_input_convolution(N, case, c, cstride):
    torch.manual_seed(7)
    h, w = 7, 65
    img = torch.randn(1, 2, h, w, device="cuda:0")
    v = torch.randn(1, h, w, cstride, device="cuda:0").bfloat16()
    v[0, 2:5, 28:33, ::2] = 0  # zero gradients around the infinity at (3, 30)
    u, pu, q, pq = case
    if u is not None:
        img[0, 1, pu[0], pu[1]] = u
    if q is not None:
        v[0, pq[0], pq[1], 0] = q
    dw, db = torch.zeros(c, 2, 9, device=v.device), torch.zeros(c, device=v.device)
    N.call("sgb_nn_conv_in_wgrad", 1, h, w, c, N.ptr(img), N.ptr(v), cstride, N.ptr(dw), N.ptr(db), N.stream_handle())
    for i in range(2):
        _same(dw[:, i], _sums(v[0, ..., :c], img[0, i], 1, True))
    _same(db[:, None], v[0, ..., :c].double().sum((0, 1))[:, None])


@pytest.mark.parametrize("case", CASES)
def test_output_convolution(N, case):
    torch.manual_seed(8)
    h, w, c = 7, 65, 32
    g = torch.randn(1, h, w, device="cuda:0")
    v = torch.randn(1, h, w, c, device="cuda:0").bfloat16()
    u, pu, q, pq = case
    if u is not None:
        g[0, pu[0], pu[1]] = u
    if q is not None:
        v[0, pq[0], pq[1], 0] = q
    W, dx = torch.randn(1, c, 3, 3, device=v.device), torch.empty(1, h, w, c, device=v.device, dtype=torch.bfloat16)
    gw, gb = torch.zeros(c, 9, device=v.device), torch.zeros(1, device=v.device)
    N.call("sgb_nn_conv_out_bwd", 1, h, w, c, N.ptr(g), N.ptr(W), N.ptr(v), c, N.ptr(dx), N.ptr(gw), N.ptr(gb),
           N.stream_handle())
    _same(gw, _sums(v[0], g[0], -1, False))
