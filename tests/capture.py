"""What a call would launch, from a captured graph; nothing is executed."""
import ctypes

import torch


class KernelParams(ctypes.Structure):  # CUDA_KERNEL_NODE_PARAMS (v2)
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("smem", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def kernel_launches(issue):
    """(grid x, block x, dynamic shared memory) of every kernel that issue(stream) enqueues."""
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
    assert cu.cuGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
    out = []
    for node in nodes:
        kind, p = ctypes.c_int(-1), KernelParams()
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        if kind.value == 0:  # CU_GRAPH_NODE_TYPE_KERNEL
            assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(p)) == 0
            out.append((p.grid[0], p.block[0], p.smem))
    assert cu.cuGraphDestroy(graph) == 0
    return out
