"""The tile kernels load coefficient rows and tables before they wait for the
launch before them; a loop's first step must therefore not be a programmatic
dependent of whatever the caller launched last (here the kernel that computes the
coefficient planes), while the later steps are.  Seen in the dependency types of a
captured graph; nothing is executed.
"""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


class EdgeData(ctypes.Structure):  # CUgraphEdgeData
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte),
                ("reserved", ctypes.c_ubyte * 5)]


DEFAULT, PROGRAMMATIC = 0, 1


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from seistorch_gb300 import _native
    _native.load(build_if_missing=False)
    return torch.device("cuda:0")


def _edge_types(issue):
    """Types of the edges of the chain that issue(stream) enqueues, in order."""
    cu = ctypes.CDLL("libcuda.so.1")
    stream = torch.cuda.Stream()
    h = ctypes.c_void_p(stream.cuda_stream)
    graph = ctypes.c_void_p()
    assert cu.cuStreamBeginCapture_v2(h, 1) == 0  # thread-local
    try:
        issue(h)
    finally:
        assert cu.cuStreamEndCapture(h, ctypes.byref(graph)) == 0
    n = ctypes.c_size_t(0)
    assert cu.cuGraphGetEdges_v2(graph, None, None, None, ctypes.byref(n)) == 0
    src, dst, data = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)(), (EdgeData * n.value)()
    assert cu.cuGraphGetEdges_v2(graph, src, dst, data, ctypes.byref(n)) == 0
    after = {src[i]: (dst[i], data[i].type) for i in range(n.value)}
    assert len(after) == n.value  # a chain
    node = (set(src) - set(dst)).pop()
    types = []
    while node in after:
        node, t = after[node]
        types.append(t)
    assert cu.cuGraphDestroy(graph) == 0
    return types


@pytest.mark.parametrize("eq,order", [("pml", 2), ("pml", 8), ("habc", 2), ("vti", 2), ("rho", 2)])
def test_first_step_waits_for_the_coefficients(dev, eq, order):
    from seistorch_gb300 import _native as N, engine
    nz, nx, B, nt = 120, 140, 2, 4
    pitch = engine.pitch_of(nx)
    plane = lambda n=1, v=1.0: torch.full((n, nz, pitch), v, device=dev)
    vp, damp, coef, rho_c = plane(1, 2000.0), plane(1, 0.0), plane(3), plane(5)
    buf = [torch.zeros(B, nz, pitch, device=dev) for _ in range(3)]
    acq = engine.Acquisition(nz, nx, [[(60, 70)]] * B, [([60], [60])] * B, torch.zeros(nt), dev)
    rec = torch.zeros(nt, B, 1, device=dev)
    g1, g = engine.grid_struct(nz, nx, pitch, 1, 0.001, 10.0), engine.grid_struct(nz, nx, pitch, B, 0.001, 10.0)
    bnd = engine.BOUNDARY_PML if eq == "pml" else engine.BOUNDARY_HABC
    m = N.AcousticModel(order, bnd, 50, 0, N.ptr(coef), N.ptr(vp), N.ptr(damp))
    q = acq.struct(rec, 1)
    bufs = N.PTR3(*[b.data_ptr() for b in buf])
    cur, prev = ctypes.c_int32(0), ctypes.c_int32(0)
    out = ctypes.byref(cur), ctypes.byref(prev)

    def issue(s):
        N.call("sgb_acoustic_coefficients", ctypes.byref(g1), N.ptr(vp), N.ptr(damp), bnd, N.ptr(coef), s)
        if eq == "vti":
            N.call("sgb_vti_forward", ctypes.byref(g), ctypes.byref(m), ctypes.byref(q), bufs, None, *out, s)
        elif eq == "rho":
            N.call("sgb_rho_forward", ctypes.byref(g), ctypes.byref(m), N.ptr(rho_c), ctypes.byref(q), bufs, None, *out, s)
        else:
            N.call("sgb_acoustic_forward", ctypes.byref(g), ctypes.byref(m), ctypes.byref(q), bufs, None, None, *out, s)

    torch.cuda.synchronize()
    assert _edge_types(issue) == [DEFAULT] + [PROGRAMMATIC] * (nt - 1)
