"""What a call launches, from its capture into a graph that never runs: the kernels' names and how many of the launches may begin
while their predecessor drains."""
import torch


def launches(call):
    """`call()` enqueues on torch's current stream; it has to have run once before (modules load on first use)."""
    from cuda.bindings import driver as d

    def ok(result):
        assert result[0] == d.CUresult.CUDA_SUCCESS, result[0]
        return result[1:]

    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        ok(d.cuStreamBeginCapture(side.cuda_stream, d.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_THREAD_LOCAL))
        try:
            call()
        finally:
            graph, = ok(d.cuStreamEndCapture(side.cuda_stream))
    try:
        _, n = ok(d.cuGraphGetNodes(graph))
        nodes, _ = ok(d.cuGraphGetNodes(graph, n))
        names = []
        for node in nodes:
            if ok(d.cuGraphNodeGetType(node))[0] != d.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
                continue
            p, = ok(d.cuGraphKernelNodeGetParams(node))
            name, = ok(d.cuFuncGetName(p.func) if int(p.func) else d.cuKernelGetName(p.kern))
            names.append(name.decode())
        *_, n = ok(d.cuGraphGetEdges_v2(graph))
        edges = ok(d.cuGraphGetEdges_v2(graph, n))[2] if n else ()
        early = sum(int(e.type) == int(d.CUgraphDependencyType.CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC) for e in edges)
    finally:
        ok(d.cuGraphDestroy(graph))
    return names, early
