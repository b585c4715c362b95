"""HABC reverse loops whose launch holds many times the tiles that are resident:
shots with one to four far tiles each (most CTAs then take tiles of the frame), with
more far tiles than CTAs that walk them, and groups of few shots.

Whole-loop gradients against the step-by-step loop under autograd (its single-step
VJP is another kernel) and against the sum of the groups' gradients.  All are fp32
restatements of the same transpose; loops of 60 steps differ by at most about
60 x 6e-8 x a few terms per cell, 2e-5 of the norm.
"""
import pytest
import torch

from tests.golden_cases import rel_l2

pytestmark = pytest.mark.gpu
W, DT, H, NT = 50, 0.001, 10.0, 60


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from seistorch_gb300 import _native
    _native.load(build_if_missing=False)
    return torch.device("cuda:0")


def _survey(nz, nx, multiple, shots, dev):
    from seistorch_gb300.habc import generate_habc_coefficients_2d
    from seistorch_gb300.utils import ricker_wave
    torch.manual_seed(nx)
    vp = (2000.0 + 800.0 * torch.rand(nz // 8 + 1, nx // 8 + 1)).repeat_interleave(8, 0).repeat_interleave(8, 1)
    vp = vp[:nz, :nx].contiguous().to(dev)
    b = generate_habc_coefficients_2d((nz, nx), W, multiple=multiple).to(dev, torch.float32)
    top = 0 if multiple else W
    src = [[(top + 2, W + 3 + (7 * s) % (nx - 2 * W - 6))] for s in range(shots)]
    rx = list(range(W, nx - W, 2))
    return vp, b, ricker_wave(30.0, DT, NT, delay=30), src, (top + 3, rx), (slice(top, nz - W), slice(W, nx - W))


@pytest.mark.parametrize("nz,nx,multiple,shots,ckpt", [(118, 312, False, 82, 0), (118, 441, False, 62, 16),
                                                       (70, 315, True, 136, 16)])
def test_gradient_with_few_far_tiles_a_shot(dev, nz, nx, multiple, shots, ckpt):
    from seistorch_gb300 import engine
    from seistorch_gb300.equations2d import acoustic_habc
    from seistorch_gb300.habc import bound_mask
    vp0, b, wav, src, (rz, rx), box = _survey(nz, nx, multiple, shots, dev)
    prop = engine.AcousticPropagator(nz, nx, DT, H, 2, "habc", W, multiple, dev)
    acq = engine.Acquisition(nz, nx, src, [([rz] * len(rx), rx)] * shots, wav, dev)
    vp = vp0.clone().requires_grad_(True)
    r, _ = engine.acoustic_loop(vp, prop, b, acq, False, ckpt)
    (r ** 2).sum().backward()
    vq = vp0.clone().requires_grad_(True)
    h1 = torch.zeros(shots, nz, nx, device=dev)
    h2 = torch.zeros_like(h1)
    masks = bound_mask(nz, nx, W, dev, shots, return_idx=True, multiple=multiple)
    sz = torch.tensor([p[0][0] for p in src], device=dev)
    sx = torch.tensor([p[0][1] for p in src], device=dev)
    loss = 0.0
    for t in range(NT):
        y, _ = acoustic_habc._time_step(vq, h1, h2, torch.tensor(DT), torch.tensor(H), b, habcs=masks)
        y = y.clone()
        y[torch.arange(shots, device=dev), sz, sx] += wav[t].to(dev)
        h2, h1 = h1, y
        loss = loss + (y[:, rz, rx] ** 2).sum()
    loss.backward()
    assert rel_l2(vp.grad[box].cpu().numpy(), vq.grad[box].cpu().numpy()) < 2e-5


@pytest.mark.parametrize("eq,order", [("habc", 2), ("habc", 4), ("habc", 6), ("habc", 8), ("born", 2), ("vti", 2),
                                      ("rho", 2)])
def test_groups_of_shots_agree(dev, eq, order):
    from seistorch_gb300 import engine
    # 34 far tiles a shot: a CTA walks several in the whole batch, one in a group of an eighth
    nz, nx, shots, groups = 251, 441, 80, 8
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    assert 34 * shots > 16 * sms > 34 * shots // groups
    vp0, b, wav, src, (rz, rx), box = _survey(nz, nx, False, shots, dev)
    par = [vp0]
    if eq == "born":
        par = [vp0 / vp0.mean() - 1.0]
    elif eq == "vti":
        par = [vp0, 0.1 * vp0 / vp0.max(), 0.05 * vp0 / vp0.max()]
    elif eq == "rho":
        par = [vp0, 310.0 * vp0 ** 0.25]

    def gradient(shot_src):
        n = len(shot_src)
        acq = engine.Acquisition(nz, nx, shot_src, [([rz] * len(rx), rx)] * n, wav, dev)
        p = [t.clone().requires_grad_(True) for t in par]
        if eq == "habc":
            r, _ = engine.acoustic_loop(p[0], engine.AcousticPropagator(nz, nx, DT, H, order, "habc", W, False, dev), b, acq)
        elif eq == "born":
            r = engine.born_loop(vp0, p[0], engine.BornPropagator(nz, nx, DT, H, order, W, False, dev), b, acq)
        elif eq == "vti":
            r = engine.vti_loop(*p, engine.VTIPropagator(nz, nx, DT, H, W, False, dev), b, acq)
        else:
            r = engine.rho_loop(*p, engine.RhoPropagator(nz, nx, DT, H, W, False, dev), b, acq)
        (r ** 2).sum().backward()
        return [t.grad[box].double().cpu().numpy() for t in p]

    whole = gradient(src)
    parts = [gradient(src[k:k + shots // groups]) for k in range(0, shots, shots // groups)]
    for i, g in enumerate(whole):
        assert rel_l2(g, sum(q[i] for q in parts)) < 2e-5
