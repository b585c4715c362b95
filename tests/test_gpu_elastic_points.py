"""Sources and receivers of the elastic reverse loop, whose corrections are
applied to the staged rows, and its saved ring: points on the rows around the
16-row bands' edges and in the corner cells of the box, several in one row,
every field as source and as receiver (vz and txz are staged one row ahead), and
widths of every remainder mod 4.

The whole-loop gradient against the step-by-step loop under autograd, whose
single-step VJP takes no points and no ring.  Both are fp32: 48 steps forward and
48 reconstructed, each rounding about five terms, give 96 x 5 x 6e-8 = 3e-5 of
the norm; the density gradient is a difference of terms about three times its
size, 1e-4.
"""
import pytest
import torch

from tests.golden_cases import rel_l2

pytestmark = pytest.mark.gpu
W = 20
FIELDS = ("vx", "vz", "txx", "tzz", "txz")


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from seistorch_gb300 import _native
    _native.load(build_if_missing=False)
    return torch.device("cuda:0")


@pytest.mark.parametrize("nx,src_type,rec_type", [(132, ["txx", "tzz"], ["vx", "vz"]), (157, ["vz"], ["vz", "txz"]),
                                                  (166, ["vx", "txz"], ["txx", "tzz", "txz", "vz"]),
                                                  (251, list(FIELDS), ["vx"])])
def test_gradient_matches_the_per_step_loop(dev, nx, src_type, rec_type):
    from seistorch_gb300 import elastic_engine, engine
    from seistorch_gb300.equations2d import elastic
    from seistorch_gb300.pml import generate_pml_coefficients_2d
    from seistorch_gb300.utils import ricker_wave
    nz, nt, dt, h = 93, 48, 0.0005, 5.0
    torch.manual_seed(nx)
    vp0 = 2500.0 + 300.0 * torch.rand(nz, nx)
    models = [m.to(dev) for m in (vp0, vp0 / 1.73, 310.0 * vp0 ** 0.25)]
    d = generate_pml_coefficients_2d((nz, nx), W).to(dev, torch.float32)
    wav = ricker_wave(40.0, dt, nt, delay=25)
    src = [[(W, W)], [(31, nx // 2), (32, nx // 2 + 1), (32, nx // 2 + 5)], [(nz - W - 1, nx - W - 1)], [(48, W + 30)]]
    zs = [W, 31, 32, 33, 47, 48, nz - W - 1]
    rec = [([z for z in zs for _ in range(3)], [W, nx // 2, nx - W - 1] * len(zs))] * len(src)
    io, nch = elastic_engine.make_io(src_type, rec_type)
    prop = elastic_engine.ElasticPropagator(nz, nx, dt, h, W, False, dev)
    acq = engine.Acquisition(nz, nx, src, rec, wav, dev)
    r, state, _ = prop.forward(*models, d, acq, io, nch, save_for_adjoint=True)
    got = prop.backward(state, acq, io, nch, 2 * r)

    leaves = [m.clone().requires_grad_(True) for m in models]
    f = [torch.zeros(len(src), nz, nx, device=dev) for _ in range(5)]
    zi, xi = torch.tensor(rec[0][0], device=dev), torch.tensor(rec[0][1], device=dev)
    loss = 0.0
    for t in range(nt):
        f = [y.clone() for y in elastic._time_step(*leaves, *f, torch.tensor(dt), torch.tensor(h), d)]
        for s, pts in enumerate(src):
            for z, x in pts:
                for n in src_type:
                    f[FIELDS.index(n)][s, z, x] += wav[t].to(dev)
        for n in rec_type:
            loss = loss + (f[FIELDS.index(n)][:, zi, xi] ** 2).sum()
    loss.backward()
    box = (slice(W, nz - W), slice(W, nx - W))
    for name, a, b in zip(("vp", "vs", "rho"), got, leaves):
        assert rel_l2(a[box].cpu().numpy(), b.grad[box].cpu().numpy()) < 1e-4, name
