"""Which kernels a call launches, read from a recorded CUDA graph through the driver (nothing is profiled)."""
import ctypes

import torch


class _KernelNode(ctypes.Structure):          # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3), ("shared", ctypes.c_uint),
                ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p), ("kern", ctypes.c_void_p), ("context", ctypes.c_void_p)]


class _EdgeData(ctypes.Structure):            # CUgraphEdgeData
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte), ("reserved", ctypes.c_ubyte * 5)]


def launched(call):
    """``[(mangled name, grid)]`` of one call, in launch order (``call`` runs once before it is recorded)."""
    return [(name, grid) for name, grid, _ in recorded(call)]


def recorded(call):
    """``[(mangled name, grid, early)]``: ``early`` where the kernel may start before the launch in front of it has ended."""
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        call()
    driver = ctypes.CDLL("libcuda.so.1")

    def check(status):
        assert status == 0, f"driver call failed with code {status}"

    handle, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    check(driver.cuGraphGetNodes(handle, None, ctypes.byref(count)))
    nodes = (ctypes.c_void_p * count.value)()
    check(driver.cuGraphGetNodes(handle, nodes, ctypes.byref(count)))
    edges = ctypes.c_size_t(0)
    check(driver.cuGraphGetEdges_v2(handle, None, None, None, ctypes.byref(edges)))
    sources, targets, data = (ctypes.c_void_p * edges.value)(), (ctypes.c_void_p * edges.value)(), (_EdgeData * edges.value)()
    if edges.value:
        check(driver.cuGraphGetEdges_v2(handle, sources, targets, data, ctypes.byref(edges)))
    early = {target for target, edge in zip(targets, data) if edge.type == 1}      # CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC
    found = []
    for node in nodes:
        kind = ctypes.c_int(-1)
        check(driver.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)))
        if kind.value != 0:                    # not a kernel
            continue
        params, name = _KernelNode(), ctypes.c_char_p()
        check(driver.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(params)))
        if params.kern:
            check(driver.cuKernelGetName(ctypes.byref(name), ctypes.c_void_p(params.kern)))
        else:
            check(driver.cuFuncGetName(ctypes.byref(name), ctypes.c_void_p(params.func)))
        found.append((name.value.decode(), tuple(params.grid), node in early))
    return found
