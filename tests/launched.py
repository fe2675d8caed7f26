"""Which kernels a call launches, and in what shape: the kernel nodes of a graph that it is captured into (nothing runs)."""
import collections
import ctypes

import torch

Launch = collections.namedtuple("Launch", "name blocks threads shared_bytes")


class _Params(ctypes.Structure):
    """cudaKernelNodeParams."""
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3), ("shared_bytes", ctypes.c_uint),
                ("kernel_params", ctypes.c_void_p), ("extra", ctypes.c_void_p)]


def launched(call):
    """The kernels that call() launches on the current stream: names as the compiler has them, blocks, threads of a block, bytes
    of dynamic shared memory.  The call runs once beforehand."""
    rt = ctypes.CDLL("libcudart.so.12")
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    raw, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t()
    assert rt.cudaGraphGetNodes(raw, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert rt.cudaGraphGetNodes(raw, nodes, ctypes.byref(count)) == 0
    out = []
    for node in nodes:
        kind, params, name = ctypes.c_int(), _Params(), ctypes.c_char_p()
        assert rt.cudaGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        if kind.value != 0:  # cudaGraphNodeTypeKernel
            continue
        assert rt.cudaGraphKernelNodeGetParams(ctypes.c_void_p(node), ctypes.byref(params)) == 0
        assert rt.cudaFuncGetName(ctypes.byref(name), ctypes.c_void_p(params.func)) == 0
        blocks, threads = (v[0] * v[1] * v[2] for v in (params.grid, params.block))
        out.append(Launch(name.value.decode(), blocks, threads, params.shared_bytes))
    return out
