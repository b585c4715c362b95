"""Receiver tables of the acoustic tile kernels: rows of more receivers than a
CTA loads at a time, wells (one receiver in each row of a band), the grid's
corners, duplicates and columns in any order, on grids whose last tile is
partial in both directions.

Records and the gradient against the fp64 oracle (the tolerances of the other
parity tests: 1e-5 and 1e-4); the order of a row's entries in the table must
not change a record at all.
"""
import numpy as np
import pytest
import torch

from oracle import adjoint, fd2d
from tests.golden_cases import rel_l2

pytestmark = pytest.mark.gpu
W = 10


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from seistorch_gb300 import _native
    _native.load(build_if_missing=False)
    return torch.device("cuda:0")


def _receivers(kind, nz, nx):
    if kind == "row":  # one full row, twice over: more than 8 x 128 table entries
        return [W + 1] * (2 * nx), list(range(nx)) * 2
    if kind == "well":  # a column through every row, and the four corners
        return list(range(nz)) + [0, 0, nz - 1, nz - 1], [W + 7] * nz + [0, nx - 1, 0, nx - 1]
    zs, xs = np.mgrid[W:nz - W:3, 0:nx:29]  # scattered over the rows of every band
    return zs.reshape(-1).tolist(), xs.reshape(-1).tolist()


@pytest.mark.parametrize("kind,nz,nx,order", [("row", 38, 533, 4), ("well", 49, 131, 8), ("grid", 33, 259, 2)])
def test_records_and_gradient(dev, kind, nz, nx, order):
    from seistorch_gb300 import engine
    vp = np.full((nz, nx), 1800.0)
    vp[nz // 2:] = 2400.0
    d = fd2d.pml_profile_2d((nz, nx), W)
    dt, h, nt = 0.001, 10.0, 50
    wav = fd2d.ricker(25.0, dt, nt, delay=40)
    zs, xs = _receivers(kind, nz, nx)
    src = [[(W + 2, W + 5)], [(nz // 2, nx // 2)]]
    rec = [(zs, xs)] * 2
    prop = engine.AcousticPropagator(nz, nx, dt, h, order, "pml", W, False, dev)
    acq = engine.Acquisition(nz, nx, src, rec, wav, dev)
    vpt = torch.tensor(vp, dtype=torch.float32, device=dev, requires_grad=True)
    dmp = torch.tensor(d, dtype=torch.float32, device=dev)
    r, illum = engine.acoustic_loop(vpt, prop, dmp, acq, True, 20)
    (r.double() ** 2).sum().backward()
    want = fd2d.forward("acoustic", {"vp": vp}, d, dt, h, wav, src, rec, order=order)
    got = r.detach().cpu().numpy().reshape(nt, 2, len(zs), 1).transpose(1, 0, 2, 3)
    assert rel_l2(got, np.stack(want["records"])) < 1e-5
    g = adjoint.acoustic_pml_gradient(vp, d, dt, h, wav, src, rec, [2 * x for x in want["records"]], order=order)
    box = (slice(W, nz - W), slice(W, nx - W))
    assert rel_l2(vpt.grad.cpu().numpy()[box], g[box]) < 1e-4
    # the same table with every row's entries in reverse order
    ptr = acq.rec_row_ptr.cpu().numpy()
    perm = np.concatenate([np.arange(a, b)[::-1] for a, b in zip(ptr[:-1], ptr[1:])]).astype(np.int64)
    perm = torch.as_tensor(perm, device=dev)
    acq.rec_x, acq.rec_col = acq.rec_x[perm].contiguous(), acq.rec_col[perm].contiguous()
    with torch.no_grad():
        r2, illum2 = engine.acoustic_loop(vpt, prop, dmp, acq, True, 20)
    assert torch.equal(r2, r.detach())
    # fp32 sums of 50 x 2 terms in another order
    assert rel_l2(illum2.cpu().numpy(), illum.cpu().numpy()) < 1e-6
