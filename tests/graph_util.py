"""Which kernels a CUDA graph launches, by the driver's graph queries."""
from __future__ import annotations

import ctypes as C

import torch


class _KernelNode(C.Structure):  # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("shared", C.c_uint),
                ("params", C.c_void_p), ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def _kernels(graph: int) -> list[tuple[str, int]]:
    cu = C.CDLL("libcuda.so.1")
    n = C.c_size_t()
    assert cu.cuGraphGetNodes(C.c_void_p(graph), None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(C.c_void_p(graph), nodes, C.byref(n)) == 0
    out = []
    for node in nodes:
        kind = C.c_int()
        assert cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        if kind.value == 0:  # a kernel
            p = _KernelNode()
            assert cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)) == 0
            name = C.c_char_p()
            if p.func:
                assert cu.cuFuncGetName(C.byref(name), C.c_void_p(p.func)) == 0
            else:
                assert cu.cuKernelGetName(C.byref(name), C.c_void_p(p.kern)) == 0
            out.append((name.value.decode(), int(p.block[0])))
    return out


def captured_kernels(call) -> list[tuple[str, int]]:
    """(mangled name, threads a block) of each kernel that call() launches on
    the current stream."""
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    return _kernels(graph.raw_cuda_graph())


def frame_kernels(graph) -> list[tuple[str, int]]:
    """The same of a captured frame (renderer.Graph): the third word of the
    library's graph object is its CUDA graph."""
    return _kernels(C.cast(graph.handle, C.POINTER(C.c_void_p))[2])
