"""Input convolution of more than 256 channels, whose weights are read from global
memory, in the launch right behind the optimiser step that writes them.

bf16 outputs: each is rounded by at most 2^-9, 2e-3 of the norm at most.
"""
import pytest
import torch
import torch.nn.functional as F

from tests.golden_cases import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [256, 264, 512])
def test_weights_of_the_launch_before(c):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from seistorch_gb300 import _native as N
    N.load(build_if_missing=False)
    torch.manual_seed(c)
    n, h, w = 2, 9, 37
    dev = torch.device("cuda:0")
    x = torch.randn(n, 2, h, w, device=dev)
    p = torch.randn(c * 19, device=dev) / 4  # 18 c weights, c biases
    out = torch.empty(n, h, w, c, device=dev, dtype=torch.bfloat16)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    for step in range(1, 6):
        g = torch.randn_like(p)
        N.call("sgb_nn_adam", p.numel(), N.ptr(p), N.ptr(g), N.ptr(m), N.ptr(v), 0.1, 0.9, 0.999, 1e-8, step, 0.0,
               N.stream_handle())
        N.call("sgb_nn_conv_in", n, h, w, c, N.ptr(x), N.ptr(p[:18 * c]), N.ptr(p[18 * c:]), N.ptr(out), c, 0,
               N.stream_handle())
        want = F.relu(F.conv2d(x.double(), p[:18 * c].double().view(c, 2, 3, 3), p[18 * c:].double(), padding=1))
        assert rel_l2(out.float().cpu().numpy(), want.permute(0, 2, 3, 1).cpu().numpy()) < 2e-3
