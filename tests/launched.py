"""Which kernels of the package a call launches, for tests of what a launcher chooses: the call is captured in a graph, whose nodes are read."""
import ctypes
import re

import torch


def _shown(mangled: bytes) -> str:
    demangle = ctypes.CDLL("libstdc++.so.6").__cxa_demangle
    demangle.restype = ctypes.c_void_p
    at = demangle(ctypes.c_char_p(mangled), None, None, ctypes.byref(ctypes.c_int()))
    return ctypes.string_at(at).decode() if at else mangled.decode()


def kernels(run):
    """The kernels' names (template arguments included) and launch parameters, in the graph's order, after a first call by itself."""
    from cuda.bindings import driver

    def ok(res):
        assert res[0] == driver.CUresult.CUDA_SUCCESS, res[0]
        return res[1]

    run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        run()
    raw = driver.CUgraph(graph.raw_cuda_graph())
    err, _, count = driver.cuGraphGetNodes(raw)
    assert err == driver.CUresult.CUDA_SUCCESS
    for node in ok(driver.cuGraphGetNodes(raw, count))[:count]:
        if ok(driver.cuGraphNodeGetType(node)) != driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        p = ok(driver.cuGraphKernelNodeGetParams(node))
        yield _shown(ok(driver.cuFuncGetName(p.func) if int(p.func) else driver.cuKernelGetName(p.kern))), p


def launched(run, pattern):
    """The parts of the kernels' names that ``pattern`` matches."""
    return {m.group(0) for name, _ in kernels(run) for m in [re.search(pattern, name)] if m}
