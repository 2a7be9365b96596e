"""The kernels that a piece of a program launches on a stream, found by capturing
it into a graph (nothing of it runs)."""
import re


def captured_kernels(stream, run):
    """[(kernel, integer and bool template arguments)] in launch order."""
    import torch
    from cuda.bindings import driver as cu

    def ok(r):
        assert r[0] == cu.CUresult.CUDA_SUCCESS, r
        return r[1:] if len(r) > 2 else r[1]

    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        run()
    raw = cu.CUgraph(graph.raw_cuda_graph())
    nodes, count = ok(cu.cuGraphGetNodes(raw, 256))
    assert count < 256
    out = []
    for node in nodes[:count]:
        if ok(cu.cuGraphNodeGetType(node)) != cu.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        p = ok(cu.cuGraphKernelNodeGetParams(node))
        name = (ok(cu.cuFuncGetName(p.func)) if int(p.func) else ok(cu.cuKernelGetName(p.kern))).decode()
        m = re.search(r"\d(k_[a-z0-9_]+)", name)
        out.append((m.group(1), tuple(int(v) for v in re.findall(r"L[ib](\d+)E", name))))
    del graph
    return out
