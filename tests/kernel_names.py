"""Which kernels a call launches: a test that is about one of several kernels checks that the choice by size takes that one."""
import torch
from cuda.bindings import driver


def _done(result):
    status, *values = result
    assert status == driver.CUresult.CUDA_SUCCESS, status
    return values


def kernels(f):
    """Mangled names of the kernels that ``f()`` launches on the current stream, in no particular order: recorded, not run (``f`` runs once before)."""
    f()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        f()
    raw = driver.CUgraph(graph.raw_cuda_graph())
    count = _done(driver.cuGraphGetNodes(raw, 0))[1]
    names = []
    for node in _done(driver.cuGraphGetNodes(raw, count))[0]:
        if _done(driver.cuGraphNodeGetType(node))[0] != driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        p, = _done(driver.cuGraphKernelNodeGetParams(node))
        name = _done(driver.cuFuncGetName(p.func) if int(p.func) else driver.cuKernelGetName(p.kern))[0]
        names.append(name.decode() if isinstance(name, bytes) else str(name))
    return names
