"""The forward's tile variants: a selected one is the one that runs, on small grids
too; without a selection the size of the grid decides; and both variants of that
rule on both sides of its line give the same records and gradients.
"""
import ctypes

import numpy as np
import pytest
import torch

from tests.capture import kernel_launches
from tests.golden_cases import rel_l2

pytestmark = pytest.mark.gpu
W, DT, H = 20, 0.001, 10.0


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from seistorch_gb300 import _native
    _native.load(build_if_missing=False)
    return torch.device("cuda:0")


@pytest.fixture(autouse=True)
def restore():
    yield
    from seistorch_gb300 import tuning
    tuning.select(tuning.AUTO, tuning.DEFAULT[1])


def _step_launch(dev, nz, nx, B, order):
    from seistorch_gb300 import _native as N, engine
    pitch = engine.pitch_of(nx)
    vp, damp = torch.full((nz, pitch), 2000.0, device=dev), torch.zeros(nz, pitch, device=dev)
    coef = torch.zeros(2, nz, pitch, device=dev)
    buf = [torch.zeros(B, nz, pitch, device=dev) for _ in range(3)]
    acq = engine.Acquisition(nz, nx, [[(30, 30)]] * B, [([30], [40])] * B, torch.zeros(1), dev)
    rec = torch.zeros(1, B, 1, device=dev)
    g = engine.grid_struct(nz, nx, pitch, B, DT, H)
    m = N.AcousticModel(order, engine.BOUNDARY_PML, 50, 0, N.ptr(coef), N.ptr(vp), N.ptr(damp))
    q = acq.struct(rec, 1)
    cur, prev = ctypes.c_int32(0), ctypes.c_int32(0)
    torch.cuda.synchronize()
    (one,) = kernel_launches(lambda s: N.call("sgb_acoustic_forward", ctypes.byref(g), ctypes.byref(m), ctypes.byref(q),
                                              N.PTR3(*[b.data_ptr() for b in buf]), None, None, ctypes.byref(cur),
                                              ctypes.byref(prev), s))
    return one


@pytest.mark.parametrize("order", [2, 8])
def test_a_selected_variant_is_the_one_that_runs(dev, order):
    from seistorch_gb300 import tuning
    nz, nx, B = 131, 261, 3
    stage = set()
    for cfg, (rows, warps, _, _) in enumerate(tuning.FWD_VARIANTS):
        tuning.select(cfg, tuning.DEFAULT[1])
        grid, block, smem = _step_launch(dev, nz, nx, B, order)
        assert grid == B * 3 * ((nz + rows - 1) // rows) and block == 32 * warps, cfg
        stage.add((grid, smem))
    assert len(stage) == len(tuning.FWD_VARIANTS)  # no two alike
    tuning.select(tuning.AUTO, tuning.DEFAULT[1])
    small = _step_launch(dev, nz, nx, B, order)
    large = _step_launch(dev, nz, nx, 64, order)
    for cfg, b, want in ((5, B, small), (4, 64, large)):
        tuning.select(cfg, tuning.DEFAULT[1])
        assert _step_launch(dev, nz, nx, b, order) == want


@pytest.mark.parametrize("order", [2, 4, 6, 8])
def test_sixteen_row_tiles_walked_by_resident_ctas(dev, order):
    """64 shots of 131 x 261: 1728 tiles of 16 rows, several per CTA through the
    two-stage ring.  Records against the float64 oracle (three shots) and, bit by
    bit, against groups of shots small enough for 8-row tiles; gradients against the
    sum of the groups', which differ by the order of at most 64 x 40 fp32 additions
    per cell: 6e-8 x sqrt(2560) = 3e-6 of the norm."""
    from oracle import fd2d
    from seistorch_gb300 import engine, tuning
    nz, nx, B, nt = 131, 261, 64, 40
    assert B * 3 * 9 > 8 * torch.cuda.get_device_properties(dev).multi_processor_count >= 16 * 3 * 9
    rng = np.random.default_rng(order)
    vp0 = 2000.0 + 500.0 * rng.random((nz, nx))
    d = fd2d.pml_profile_2d((nz, nx), W)
    wav = fd2d.ricker(25.0, DT, nt, delay=15)
    src = [[(W + 2 + s % 50, W + 3 + (5 * s) % 210)] for s in range(B)]
    rx = list(range(W, nx - W, 3))
    rec = [([W + 5 + s % 60] * len(rx), rx) for s in range(B)]
    prop = engine.AcousticPropagator(nz, nx, DT, H, order, "pml", W, False, dev)
    dt = torch.tensor(d, dtype=torch.float32, device=dev)

    def run(lo, hi):
        acq = engine.Acquisition(nz, nx, src[lo:hi], rec[lo:hi], wav, dev)
        vp = torch.tensor(vp0, dtype=torch.float32, device=dev, requires_grad=True)
        r, _ = engine.acoustic_loop(vp, prop, dt, acq, False, 16)
        (r ** 2).sum().backward()
        return r.detach().cpu().numpy().reshape(nt, hi - lo, len(rx)), vp.grad.double().cpu().numpy()

    parts = [run(k, k + 16) for k in range(0, B, 16)]
    want = fd2d.forward("acoustic", {"vp": vp0}, d, DT, H, wav, src[::31], rec[::31], order=order)
    for cfg in (tuning.AUTO, 4):
        tuning.select(cfg, tuning.DEFAULT[1])
        r, g = run(0, B)
        assert np.array_equal(r, np.concatenate([p[0] for p in parts], 1))
        for i, s in enumerate(range(0, B, 31)):
            assert rel_l2(r[:, s], want["records"][i].reshape(nt, len(rx))) < 1e-5
        assert rel_l2(g, sum(p[1] for p in parts)) < 3e-6
