"""What a captured CUDA graph holds: its kernels' names and the parameters that they were launched with, in the order of their capture."""

import ctypes

import numpy as np
import torch


class _KernelNode(ctypes.Structure):
    _fields_ = [("func", ctypes.c_void_p), ("sizes", ctypes.c_uint * 7), ("params", ctypes.POINTER(ctypes.c_void_p)), ("extra", ctypes.c_void_p),
                ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def capture(work):
    work()  # plans and kernel attributes outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        work()
    graph.instantiate()
    return graph


def kernels(graph):
    """(name, parameter) of each kernel; parameter(i) is the i-th one's bytes as int32 words."""
    cuda, handle, n = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert cuda.cuGraphGetNodes(handle, None, ctypes.byref(n)) == 0
    nodes, found = (ctypes.c_void_p * n.value)(), []
    assert cuda.cuGraphGetNodes(handle, nodes, ctypes.byref(n)) == 0
    for node in nodes:
        kind, k, name = ctypes.c_int(), _KernelNode(), ctypes.c_char_p()
        assert cuda.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        if kind.value != 0:  # no kernel
            continue
        assert cuda.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(k)) == 0
        of, which = ("Func", k.func) if k.func else ("Kernel", k.kern)
        assert getattr(cuda, f"cu{of}GetName")(ctypes.byref(name), ctypes.c_void_p(which)) == 0

        def parameter(i, k=k, of=of, which=which):
            at, size = ctypes.c_size_t(), ctypes.c_size_t()
            assert getattr(cuda, f"cu{of}GetParamInfo")(ctypes.c_void_p(which), ctypes.c_size_t(i), ctypes.byref(at), ctypes.byref(size)) == 0
            return np.frombuffer(ctypes.string_at(k.params[i], size.value), dtype=np.int32)
        found.append((name.value.decode(), parameter))
    return found
