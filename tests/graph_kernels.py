"""The kernels that a call launches, by name: the call is captured into a CUDA graph and the graph's nodes are read back."""


def kernels(call):
    import torch
    from cuda.bindings import driver as cu

    def ok(result):
        assert result[0] == cu.CUresult.CUDA_SUCCESS, result[0]
        return result[1]

    call()                                                      # whatever a first call sets up
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    raw = cu.CUgraph(graph.raw_cuda_graph())
    count = cu.cuGraphGetNodes(raw, 0)[2]
    names = []
    for node in ok(cu.cuGraphGetNodes(raw, count)[:2])[:count]:
        if ok(cu.cuGraphNodeGetType(node)) == cu.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            p = ok(cu.cuGraphKernelNodeGetParams(node))
            names.append(ok(cu.cuFuncGetName(p.func) if int(p.func) else cu.cuKernelGetName(p.kern)).decode())
    return names
