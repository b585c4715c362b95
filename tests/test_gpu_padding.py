"""Columns nx .. pitch - 1 of the model and coefficient planes hold no data: with
NaN there (a caller's uninitialised plane) the records and gradients of every loop
are those of zero padding.  Widths of every remainder mod 4.

Both sides run the same kernels on the same data; the gradients differ by the
order of the reduction atomics only, below 1e-6 of the norm.
"""
import numpy as np
import pytest
import torch

from tests.golden_cases import rel_l2

pytestmark = pytest.mark.gpu
W, DT, H, NT = 50, 0.001, 10.0, 50


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from seistorch_gb300 import _native
    _native.load(build_if_missing=False)
    return torch.device("cuda:0")


def _nan_pitched(a, pitch, dtype=torch.float32):
    out = torch.full((*a.shape[:-1], pitch), float("nan"), dtype=dtype, device=a.device)
    out[..., :a.shape[-1]] = a
    return out


def _run(eq, order, nz, nx, planes, dev):
    """Records and gradients of two shots near the corners."""
    from seistorch_gb300 import elastic_engine, engine
    from seistorch_gb300.habc import generate_habc_coefficients_2d
    from seistorch_gb300.pml import generate_pml_coefficients_2d
    from seistorch_gb300.utils import ricker_wave
    torch.manual_seed(nx)
    vp = (2000.0 + 800.0 * torch.rand(nz, nx)).to(dev)
    make = generate_pml_coefficients_2d if eq in ("pml", "elastic") else generate_habc_coefficients_2d
    d = make((nz, nx), W).to(dev, torch.float32)
    rx = list(range(W, nx - W))
    src = [[(W + 2, W + 1)], [(nz - W - 2, nx - W - 2)]]
    acq = engine.Acquisition(nz, nx, src, [([W + 3] * len(rx), rx)] * 2, ricker_wave(30.0, DT, NT, delay=20), dev)
    leaf = lambda t: t.clone().requires_grad_(True)
    if eq in ("pml", "habc"):
        prop = engine.AcousticPropagator(nz, nx, DT, H, order, eq, W, False, dev)
        if not planes:  # a caller's store without the share planes
            r, state, _ = prop.forward(vp, d, acq, save_for_adjoint=True)
            state.bs.habc_planes = None
            return r, [prop.backward(state, acq, 2 * r)]
        p = [leaf(vp)]
        r, _ = engine.acoustic_loop(p[0], prop, d, acq)
    elif eq == "born":
        p = [leaf(0.1 * (vp / 2400.0 - 1.0))]
        r = engine.born_loop(vp, p[0], engine.BornPropagator(nz, nx, DT, H, order, W, False, dev), d, acq)
    elif eq == "vti":
        p = [leaf(vp), leaf(4e-5 * vp), leaf(2e-5 * vp)]
        r = engine.vti_loop(*p, engine.VTIPropagator(nz, nx, DT, H, W, False, dev), d, acq)
    elif eq == "rho":
        p = [leaf(vp), leaf(310.0 * vp ** 0.25)]
        r = engine.rho_loop(*p, engine.RhoPropagator(nz, nx, DT, H, W, False, dev), d, acq)
    elif eq == "vac":
        p = [leaf(vp), leaf(vp / 40.0)]
        r = engine.vacoustic_records(*p, engine.VacousticPropagator(nz, nx, DT, H, order, W, False, dev), d, acq)
    else:
        p = [leaf(vp), leaf(vp / 1.73), leaf(310.0 * vp ** 0.25)]
        io, nch = elastic_engine.make_io(["txx", "tzz"], ["vx", "vz"])
        r, _ = elastic_engine.elastic_records(*p, elastic_engine.ElasticPropagator(nz, nx, DT, H, W, False, dev), d, acq,
                                              io, nch, False, 0)
    (r ** 2).sum().backward()
    return r.detach(), [t.grad for t in p]


@pytest.mark.parametrize("nx", [133, 134, 135])
@pytest.mark.parametrize("eq,order,planes", [("pml", 4, True), ("habc", 2, True), ("habc", 2, False), ("habc", 8, True),
                                             ("born", 2, True), ("vti", 2, True), ("rho", 2, True), ("vac", 2, True),
                                             ("elastic", 2, True)])
def test_padding_is_never_data(dev, monkeypatch, eq, order, planes, nx):
    from seistorch_gb300 import elastic_engine, engine
    want, gw = _run(eq, order, 113, nx, planes, dev)
    monkeypatch.setattr(engine, "to_pitched", _nan_pitched)
    monkeypatch.setattr(elastic_engine, "to_pitched", _nan_pitched)
    got, gg = _run(eq, order, 113, nx, planes, dev)
    assert np.array_equal(got.cpu().numpy(), want.cpu().numpy())
    for a, b in zip(gg, gw):
        assert torch.isfinite(a).all()
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 1e-6


def test_a_cell_without_a_share_takes_no_part(dev):
    """An infinite residual just outside the left strip: one reverse step later its
    right neighbour holds the stencil's infinity, not 0 x inf of a one-way line
    that does not reach it."""
    import ctypes
    from seistorch_gb300 import _native as N
    from seistorch_gb300 import engine
    from seistorch_gb300.habc import generate_habc_coefficients_2d
    nz, nx, nt, z = 120, 140, 3, 60
    vp = torch.full((nz, nx), 2000.0, device=dev)
    b = generate_habc_coefficients_2d((nz, nx), W).to(dev, torch.float32)
    prop = engine.AcousticPropagator(nz, nx, DT, H, 2, "habc", W, False, dev)
    acq = engine.Acquisition(nz, nx, [[(z, 70)]], [([z], [W])], torch.zeros(nt), dev)
    _, state, _ = prop.forward(vp, b, acq, save_for_adjoint=True)
    resid = torch.zeros(nt, 1, 1, device=dev)
    resid[2] = float("inf")
    field = lambda: torch.zeros(1, nz, prop.pitch, device=dev)
    lb, gs, gv = [field() for _ in range(3)], field(), torch.zeros(nz, prop.pitch, device=dev)
    g, q = prop.grid(1), acq.struct(resid, 1)
    N.call("sgb_acoustic_backward", ctypes.byref(g), ctypes.byref(state.model), ctypes.byref(q), ctypes.byref(state.bs),
           N.PTR3(*[t.data_ptr() for t in state.buf]), state.cur, state.prev, N.PTR3(*[t.data_ptr() for t in lb]),
           N.ptr(gs), N.ptr(gv), N.stream_handle())
    # La_3 (the residual alone) and La_2 are the two written last
    la3 = [t for t in lb if torch.isinf(t).sum() == 1 and not torch.isnan(t).any()]
    la2 = [t for t in lb if torch.isinf(t).sum() > 1]
    assert len(la3) == 1 and len(la2) == 1 and torch.isinf(la3[0][0, z, W])
    a = la2[0][0]
    nan = torch.isnan(a)
    nan[z, W] = False
    assert not nan.any()
    assert torch.isinf(a[z, W + 1]) and torch.isinf(a[z + 1, W])
