"""Tiles of the HABC reverse step near the left and right strips, where a lane
takes four columns at once: widths of every remainder mod 4, grids without and
with tiles out of reach of the strips, with and without a top strip, and the
shares from planes or evaluated in the kernel.

The whole-loop gradient against the step-by-step loop under autograd, whose
single-step VJP is another kernel (a gather per cell).  Both are fp32
restatements of the same transpose; two such loops of 60 steps differ by at most
about 60 x 6e-8 x a few terms per cell, 2e-5 of the norm.
"""
import pytest
import torch

from tests.golden_cases import rel_l2

pytestmark = pytest.mark.gpu
W = 50


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from seistorch_gb300 import _native
    _native.load(build_if_missing=False)
    return torch.device("cuda:0")


@pytest.mark.parametrize("planes", [True, False])
@pytest.mark.parametrize("nz,nx,multiple", [(112, 131, False), (109, 134, True), (150, 421, False), (131, 399, True)])
def test_gradient_matches_the_per_step_loop(dev, nz, nx, multiple, planes):
    from seistorch_gb300 import engine
    from seistorch_gb300.equations2d import acoustic_habc
    from seistorch_gb300.habc import bound_mask, generate_habc_coefficients_2d
    from seistorch_gb300.utils import ricker_wave
    dt, h, nt = 0.001, 10.0, 60
    torch.manual_seed(nx)
    vp0 = (2000.0 + 800.0 * torch.rand(nz // 8 + 1, nx // 8 + 1)).repeat_interleave(8, 0).repeat_interleave(8, 1)
    vp0 = vp0[:nz, :nx].contiguous().to(dev)
    b = generate_habc_coefficients_2d((nz, nx), W, multiple=multiple).to(dev, torch.float32)
    top = 0 if multiple else W
    wav = ricker_wave(30.0, dt, nt, delay=30)
    src = [[(top + 2, W + 3)], [(nz - W - 2, nx - W - 4)]]  # close to the strips
    rx = list(range(W, nx - W, 2))
    rec = [([top + 3] * len(rx), rx)] * 2
    prop = engine.AcousticPropagator(nz, nx, dt, h, 2, "habc", W, multiple, dev)
    acq = engine.Acquisition(nz, nx, src, rec, wav, dev)
    vp = vp0.clone().requires_grad_(True)
    if planes:
        r, _ = engine.acoustic_loop(vp, prop, b, acq)
        (r ** 2).sum().backward()
        got = vp.grad
    else:  # a C caller's store without the planes
        r, state, _ = prop.forward(vp0, b, acq, save_for_adjoint=True)
        state.bs.habc_planes = None
        got = prop.backward(state, acq, 2 * r)
    # the same loop, step by step
    vq = vp0.clone().requires_grad_(True)
    h1 = torch.zeros(2, nz, nx, device=dev)
    h2 = torch.zeros_like(h1)
    masks = bound_mask(nz, nx, W, dev, 2, return_idx=True, multiple=multiple)
    loss = 0.0
    for t in range(nt):
        y, _ = acoustic_habc._time_step(vq, h1, h2, torch.tensor(dt), torch.tensor(h), b, habcs=masks)
        y = y.clone()
        for s, pts in enumerate(src):
            y[s, pts[0][0], pts[0][1]] += wav[t].to(dev)
        h2, h1 = h1, y
        loss = loss + (y[:, top + 3, rx] ** 2).sum()
    loss.backward()
    box = (slice(top, nz - W), slice(W, nx - W))
    assert rel_l2(got[box].cpu().numpy(), vq.grad[box].cpu().numpy()) < 2e-5


@pytest.mark.parametrize("nz,nx,multiple", [(112, 131, False), (109, 134, True), (131, 401, False), (107, 264, True),
                                            (121, 92, False)])
def test_forward_matches_the_per_step_loop(dev, nz, nx, multiple):
    """Corners where four columns lie on one side, on a diagonal or on two
    sides (every remainder of the width mod 4, and a grid narrower than two
    strips), against the per-step kernel, which takes every cell by itself: the
    last field over the whole grid.  60 steps of fp32 rounding, 2e-5 of the norm."""
    from seistorch_gb300 import engine
    from seistorch_gb300.equations2d import acoustic_habc
    from seistorch_gb300.habc import bound_mask, generate_habc_coefficients_2d
    from seistorch_gb300.utils import ricker_wave
    dt, h, nt = 0.001, 10.0, 60
    torch.manual_seed(nx)
    vp = (2000.0 + 800.0 * torch.rand(nz, nx)).to(dev)
    b = generate_habc_coefficients_2d((nz, max(nx, 2 * W)), W, multiple=multiple)[:, :nx].contiguous()
    b = b.to(dev, torch.float32)
    wav = ricker_wave(30.0, dt, nt, delay=30)
    src = [[(5, 7)], [(nz - 8, nx - 6)], [(4, nx - 9)], [(nz - 5, 6)]]  # one in every corner
    acq = engine.Acquisition(nz, nx, src, [([nz // 2], [nx // 2])] * 4, wav, dev)
    prop = engine.AcousticPropagator(nz, nx, dt, h, 2, "habc", W, multiple, dev)
    _, state, _ = prop.forward(vp, b, acq)
    got = state.buf[state.cur]
    h1 = torch.zeros(4, nz, nx, device=dev)
    h2 = torch.zeros_like(h1)
    masks = bound_mask(nz, nx, W, dev, 4, return_idx=True, multiple=multiple)
    for t in range(nt):
        y, _ = acoustic_habc._time_step(vp, h1, h2, torch.tensor(dt), torch.tensor(h), b, habcs=masks)
        y = y.clone()
        for s, pts in enumerate(src):
            y[s, pts[0][0], pts[0][1]] += wav[t].to(dev)
        h2, h1 = h1, y
    assert rel_l2(got[..., :nx].cpu().numpy(), h1.cpu().numpy()) < 2e-5
