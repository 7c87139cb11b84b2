"""The kernels that a call launches: the call is captured into a CUDA graph and the graph's nodes are read back."""


def _ok(result):
    from cuda.bindings import driver as cu
    assert result[0] == cu.CUresult.CUDA_SUCCESS, result[0]
    return result[1]


def _kernel_nodes(call):
    import torch
    from cuda.bindings import driver as cu
    call()                                                      # whatever a first call sets up
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    raw = cu.CUgraph(graph.raw_cuda_graph())
    count = cu.cuGraphGetNodes(raw, 0)[2]
    nodes = _ok(cu.cuGraphGetNodes(raw, count)[:2])[:count]
    return graph, [_ok(cu.cuGraphKernelNodeGetParams(n)) for n in nodes if _ok(cu.cuGraphNodeGetType(n)) == cu.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL]


def kernels(call):
    """The kernels' names."""
    from cuda.bindings import driver as cu
    _graph, nodes = _kernel_nodes(call)
    return [_ok(cu.cuFuncGetName(p.func) if int(p.func) else cu.cuKernelGetName(p.kern)).decode() for p in nodes]


def dynamic_shared_memory_limits(call):
    """The dynamic shared memory that each of the library's kernels in the call is allowed."""
    from cuda.bindings import driver as cu
    _graph, nodes = _kernel_nodes(call)
    functions = [p.func if int(p.func) else _ok(cu.cuKernelGetFunction(p.kern)) for p in nodes]
    return [_ok(cu.cuFuncGetAttribute(cu.CUfunction_attribute.CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, f)) for f in functions
            if "b200rl" in _ok(cu.cuFuncGetName(f)).decode()]
