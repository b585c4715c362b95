"""Weight and bias gradients of the preconditioner's convolutions from NHWC
tensors against PyTorch: the tensor-core kernel at channel counts below, at and
above its panels (64 input channels, 32 / 64 / 128 output channels per tile),
one pixel chunk to many splits, and the input / output convolutions' kernel at
ragged image sizes and channel counts.

Operands are bf16, sums fp32: an fp32 sum of P products in another order is off
by about eps sqrt(P) relative to the norm of the result, below 1e-5 for the
1e5 pixels used here (products of bf16 are exact).
"""
import ctypes

import pytest
import torch
import torch.nn.functional as F

from tests.golden_cases import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def N():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from seistorch_gb300 import _native
    _native.load(build_if_missing=False)
    return _native


def _bf16(*shape):
    return torch.randn(*shape, device="cuda:0").bfloat16()


def _wgrad64(x, dy):
    """dL/dW of a 3x3 convolution, padding 1, in float64 (NHWC operands)."""
    n, h, w, ci = x.shape
    xp = F.pad(x.double(), (0, 0, 1, 1, 1, 1))
    g = dy.double().reshape(-1, dy.shape[-1])
    taps = [g.T @ xp[:, ky:ky + h, kx:kx + w].reshape(-1, ci) for ky in range(3) for kx in range(3)]
    return torch.stack(taps, -1)  # (cout, cin, 9)


@pytest.mark.parametrize("n,h,w,cin,cout", [(1, 1, 64, 8, 8), (2, 8, 128, 32, 32), (1, 16, 64, 64, 32),
                                            (1, 3, 192, 72, 64), (2, 5, 64, 96, 40), (1, 4, 128, 128, 256),
                                            (1, 2, 64, 200, 136), (3, 40, 512, 96, 32)])
def test_weight_and_bias_gradient_nhwc(N, n, h, w, cin, cout):
    torch.manual_seed(cin * 1000 + cout)
    x, dy = _bf16(n, h, w, cin), _bf16(n, h, w, cout)
    dw = torch.ones(cout, cin, 9, device=x.device)
    db = torch.ones(cout, device=x.device)
    p = N.NnWgradNhwc(n, h, w, cin, cout, N.ptr(dy), N.ptr(x), N.ptr(dw))
    N.call("sgb_nn_conv3x3_wgrad_nhwc", ctypes.byref(p), N.stream_handle())
    N.call("sgb_nn_bias_grad_nhwc", n * h * w, cout, N.ptr(dy), N.ptr(db), N.stream_handle())
    want = 1.0 + _wgrad64(x, dy)
    assert rel_l2(dw.cpu().numpy(), want.cpu().numpy()) < 1e-5
    assert rel_l2(db.cpu().numpy(), (1.0 + dy.double().sum((0, 1, 2))).cpu().numpy()) < 1e-5
    assert N.device_status() == 0


@pytest.mark.parametrize("n,h,w,c,cstride", [(2, 33, 70, 32, 32), (1, 16, 64, 8, 24), (1, 5, 3, 40, 40),
                                             (1, 7, 65, 5, 11)])
def test_input_and_output_convolution_weight_gradients(N, n, h, w, c, cstride):
    torch.manual_seed(h * w + c)
    v = _bf16(n, h, w, cstride)
    img = torch.randn(n, 2, h, w, device=v.device)
    dw, db = torch.zeros(c, 2, 9, device=v.device), torch.zeros(c, device=v.device)
    N.call("sgb_nn_conv_in_wgrad", n, h, w, c, N.ptr(img), N.ptr(v), cstride, N.ptr(dw), N.ptr(db),
           N.stream_handle())
    dy = v[..., :c]
    assert rel_l2(dw.cpu().numpy(), _wgrad64(img.permute(0, 2, 3, 1), dy).cpu().numpy()) < 1e-5
    assert rel_l2(db.cpu().numpy(), dy.double().sum((0, 1, 2)).cpu().numpy()) < 1e-5
    if c % 8 or cstride % 8:
        return
    W = torch.randn(1, c, 3, 3, device=v.device)
    dx = torch.empty(n, h, w, c, device=v.device, dtype=torch.bfloat16)
    gw, gb = torch.zeros(c, 9, device=v.device), torch.zeros(1, device=v.device)
    g = img[:, 0].contiguous()
    N.call("sgb_nn_conv_out_bwd", n, h, w, c, N.ptr(g), N.ptr(W), N.ptr(v), cstride, N.ptr(dx), N.ptr(gw), N.ptr(gb),
           N.stream_handle())
    want = _wgrad64(dy, g[..., None])[0]
    assert rel_l2(gw.cpu().numpy(), want.cpu().numpy()) < 1e-5
    assert abs(gb.item() - g.double().sum().item()) < 1e-5 * g.double().abs().sum().item()
