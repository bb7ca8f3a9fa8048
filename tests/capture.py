"""What a library call launches, read from the CUDA graph that its stream captures."""
import ctypes

import pytest


class _Edge(ctypes.Structure):  # CUgraphEdgeData
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte),
                ("reserved", ctypes.c_ubyte * 5)]


def captured(plan, call):
    """(grid x sizes of the kernels, edge types: 1 where a kernel may start before its predecessor has
    ended) of one call of call() on `plan`, whose work fields have been allocated by an earlier call"""
    import torch
    cu = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert r[0] == cu.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else r[1:]

    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    plan.set_stream(stream)
    ok(cu.cuStreamBeginCapture(stream.cuda_stream, cu.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED))
    call()
    graph = ok(cu.cuStreamEndCapture(stream.cuda_stream))
    nodes, n = ok(cu.cuGraphGetNodes(graph, 1024))
    kernel = cu.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL
    grids = [ok(cu.cuGraphKernelNodeGetParams(v)).gridDimX for v in nodes[:n] if ok(cu.cuGraphNodeGetType(v)) == kernel]
    count, ends, edges = ctypes.c_size_t(1024), (ctypes.c_void_p * 2048)(), (_Edge * 1024)()
    rc = ctypes.CDLL("libcuda.so.1").cuGraphGetEdges_v2(ctypes.c_void_p(int(graph)), ends, ctypes.byref(ends, 8192), edges,
                                                        ctypes.byref(count))
    assert rc == 0 and count.value < 1024
    types = [e.type for e in edges[:count.value]]
    ok(cu.cuGraphDestroy(graph))
    plan.set_stream(torch.cuda.current_stream())
    return grids, types
