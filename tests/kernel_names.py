"""What a call launches: the nodes of a CUDA graph that captures it."""
import ctypes

KERNEL = 0  # CUgraphNodeType


class _KernelParams(ctypes.Structure):  # CUDA_KERNEL_NODE_PARAMS
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3),
                ("shared", ctypes.c_uint), ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def launches(call):
    """[(node type, kernel name as the linker knows it, blocks, threads per block)] of
    ``call()``, captured on a stream of its own and not run (name None: not a kernel)."""
    import torch
    cu = ctypes.CDLL("libcuda.so.1")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        call()
    raw, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t()
    assert cu.cuGraphGetNodes(raw, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert cu.cuGraphGetNodes(raw, nodes, ctypes.byref(count)) == 0
    found = []
    for n in nodes:
        t = ctypes.c_int()
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(n), ctypes.byref(t)) == 0
        if t.value != KERNEL:
            found.append((t.value, None, 0, 0))
            continue
        p, name = _KernelParams(), ctypes.c_char_p()
        assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(n), ctypes.byref(p)) == 0
        get = (cu.cuKernelGetName, p.kern) if p.kern else (cu.cuFuncGetName, p.func)
        assert get[0](ctypes.byref(name), ctypes.c_void_p(get[1])) == 0
        found.append((KERNEL, name.value.decode(), p.grid[0], p.block[0]))
    return found


def captured(call):
    """(node types, kernel names) of ``call()``."""
    found = launches(call)
    return [f[0] for f in found], [f[1] for f in found if f[1]]
