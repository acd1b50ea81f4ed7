"""Which kernels a call launches, read from a capture of it: nothing runs."""
import ctypes

import torch
from cuda.bindings import driver


class _EdgeData(ctypes.Structure):  # CUgraphEdgeData
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte), ("reserved", ctypes.c_ubyte * 5)]


PROGRAMMATIC = driver.CUgraphDependencyType.CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC.value


def _ok(result):
    assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
    return result[1:]


def _edges(raw):
    """(from, to, type) of every edge.  Through ctypes: the bindings' edge data does not outlive the call that returns it."""
    get = ctypes.CDLL("libcuda.so.1").cuGraphGetEdges_v2
    get.argtypes = [ctypes.c_void_p] * 5
    count = ctypes.c_size_t(0)
    assert get(raw, None, None, None, ctypes.byref(count)) == 0
    n = count.value
    sources, targets, data = (ctypes.c_void_p * n)(), (ctypes.c_void_p * n)(), (_EdgeData * n)()
    assert n == 0 or get(raw, sources, targets, data, ctypes.byref(count)) == 0
    return [(sources[i], targets[i], data[i].type) for i in range(n)]


def launches(*calls):
    """The kernels of the calls, captured one after the other on one stream, as (name, early) in their order; early: the kernel may
    start before the one ahead of it has ended (programmatic stream serialization).  Each call has to have run once before, so that
    the buffers it keeps are there."""
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        for call in calls:
            call()
    raw = graph.raw_cuda_graph()
    nodes, count = _ok(driver.cuGraphGetNodes(driver.CUgraph(raw)))
    nodes, _ = _ok(driver.cuGraphGetNodes(driver.CUgraph(raw), count))
    before = {t: (s, kind) for s, t, kind in _edges(raw)}
    names = {}
    for node in nodes:
        kind, = _ok(driver.cuGraphNodeGetType(node))
        if kind == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            params, = _ok(driver.cuGraphKernelNodeGetParams(node))
            name, = _ok(driver.cuFuncGetName(params.func)) if int(params.func) else _ok(driver.cuKernelGetName(params.kern))
            names[int(node)] = name.decode()

    def place(node):  # (each has one predecessor at most, on one stream)
        return 1 + place(before[node][0]) if node in before else 0

    return [(names[n], n in before and before[n][1] == PROGRAMMATIC) for n in sorted(names, key=place)]


def kernels(*calls):
    """The kernels' plain names."""
    known = ("resident_kernel", "stream_kernel", "exact_kernel", "tile_cluster_kernel", "tile_run_kernel", "batch_kernel", "umma_kernel")
    return [next((k for k in known if k in name), name) for name, _ in launches(*calls)]
