"""What a call launches: (kernel name, CTAs) of every kernel it puts on a stream, from a capture that never runs."""
import ctypes

import torch

RELAXED = 2  # CU_STREAM_CAPTURE_MODE_RELAXED
KERNEL = 0   # CU_GRAPH_NODE_TYPE_KERNEL


class KernelNode(ctypes.Structure):
    """CUDA_KERNEL_NODE_PARAMS (v2)."""
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("smem", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def launches(call):
    """call(stream) is made once as it is, then once in a capture; the kernels of the latter."""
    cu = ctypes.CDLL("libcuda.so.1")
    p = ctypes.c_void_p

    def ok(rc):
        assert rc == 0, "CUDA driver error %d" % rc

    st = torch.cuda.Stream()
    call(st)
    torch.cuda.synchronize()
    graph = p()
    ok(cu.cuStreamBeginCapture_v2(p(st.cuda_stream), RELAXED))
    try:
        call(st)
    finally:
        ok(cu.cuStreamEndCapture(p(st.cuda_stream), ctypes.byref(graph)))
    n = ctypes.c_size_t()
    ok(cu.cuGraphGetNodes(graph, None, ctypes.byref(n)))
    nodes = (p * n.value)()
    ok(cu.cuGraphGetNodes(graph, nodes, ctypes.byref(n)))
    out = []
    for node in nodes:
        kind = ctypes.c_int()
        ok(cu.cuGraphNodeGetType(p(node), ctypes.byref(kind)))
        if kind.value != KERNEL:
            continue
        k = KernelNode()
        name = ctypes.c_char_p()
        ok(cu.cuGraphKernelNodeGetParams_v2(p(node), ctypes.byref(k)))
        if k.func:
            ok(cu.cuFuncGetName(ctypes.byref(name), p(k.func)))
        else:
            ok(cu.cuKernelGetName(ctypes.byref(name), p(k.kern)))
        out.append((name.value.decode(), k.grid[0] * k.grid[1] * k.grid[2]))
    ok(cu.cuGraphDestroy(graph))
    return out
