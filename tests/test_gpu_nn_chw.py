"""Bias gradient from a channel-major copy (sgb_nn_to_chw, sgb_nn_bias_grad) against
PyTorch in float64: bf16 summands, fp32 sums of at most 12 k terms, below
eps sqrt(12000) = 7e-6 of the sum of magnitudes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w,c", [(1, 1, 64, 8), (3, 33, 70, 40), (2, 48, 128, 136)])
def test_bias_gradient_from_chw(n, h, w, c):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from seistorch_gb300 import _native as N
    N.load(build_if_missing=False)
    torch.manual_seed(c)
    dy = torch.randn(n, h, w, c, device="cuda:0").bfloat16()
    chw = torch.empty(n, c, h, w, device=dy.device, dtype=torch.bfloat16)
    db = torch.ones(c, device=dy.device)
    N.call("sgb_nn_to_chw", n, h, w, c, c, 0, N.ptr(dy), 1, N.ptr(chw), N.stream_handle())
    N.call("sgb_nn_bias_grad", n, h * w, c, N.ptr(chw), N.ptr(db), N.stream_handle())
    assert torch.equal(chw, dy.permute(0, 3, 1, 2))
    d = dy.double()
    assert ((db.double() - 1.0 - d.sum((0, 1, 2))).abs() <= 7e-6 * (1.0 + d.abs().sum((0, 1, 2)))).all()
