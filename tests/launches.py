"""The kernels that a call launches, from its CUDA graph."""
import re

import torch


def _short(mangled):
    """split_rows<1> for the split_rows_kernel of a single template argument `true`, without namespaces and the rest."""
    name, vector = re.search(r".*\d([a-z][a-z_]*\d*)_kernel(?:ILb([01])EE)?", mangled).groups()
    if "TransposedProblem" in mangled:
        name += "_transposed"
    return name + ("<%s>" % vector if vector else "")


def kernels(fn):
    """Short names of the kernels that fn launches, in the order of the graph's nodes."""
    from cuda.bindings import driver
    fn()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        fn()
    graph = driver.CUgraph(g.raw_cuda_graph())
    _, _, count = driver.cuGraphGetNodes(graph)
    _, nodes, _ = driver.cuGraphGetNodes(graph, count)
    names = []
    for n in nodes[:count]:
        if driver.cuGraphNodeGetType(n)[1] == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            params = driver.cuGraphKernelNodeGetParams(n)[1]
            status, name = driver.cuFuncGetName(params.func)
            assert status == driver.CUresult.CUDA_SUCCESS, status
            names.append(_short(name.decode()))
    return names
