"""Which kernels a call launches, by name: read from a graph that it is captured into."""

import torch
from cuda.bindings import driver


def _ok(result):
    assert result[0] == driver.CUresult.CUDA_SUCCESS, result
    return result[1:]


def kernel_names(call):
    """The names, as the compiler made them, in the order of launch. ``call`` runs once before it is captured."""
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    raw = graph.raw_cuda_graph()
    count = _ok(driver.cuGraphGetNodes(raw))[-1]
    names = []
    for node in _ok(driver.cuGraphGetNodes(raw, count))[0]:
        if _ok(driver.cuGraphNodeGetType(node))[0] == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            names.append(_ok(driver.cuFuncGetName(_ok(driver.cuGraphKernelNodeGetParams(node))[0].func))[0].decode())
    return names
