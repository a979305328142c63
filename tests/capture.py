"""What a call launches: the call is captured into a CUDA graph (nothing runs) and the graph is read."""
import collections

import torch
from cuda.bindings import driver as cu

# name, CTAs of the grid, bytes of dynamic shared memory; `overlaps`: the name of the kernel whose end this launch may
# overlap (a programmatic edge), or None
Launch = collections.namedtuple("Launch", "name grid smem overlaps")


def _ok(result):
    assert result[0] == cu.CUresult.CUDA_SUCCESS, result[0]
    return result[1] if len(result) == 2 else result[1:]


def launches(ctx, call):
    """The kernels that call() puts into the context's stream, in order."""
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    try:
        _ok(cu.cuStreamBeginCapture(stream.cuda_stream, cu.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_RELAXED))
        try:
            call()
        finally:
            ended = cu.cuStreamEndCapture(stream.cuda_stream)
    finally:
        ctx.set_stream(0)
    graph = _ok(ended)
    nodes, count = _ok(cu.cuGraphGetNodes(graph, 0))
    nodes, count = _ok(cu.cuGraphGetNodes(graph, count))
    froms, tos, data, count = _ok(cu.cuGraphGetEdges_v2(graph, 0))
    froms, tos, data, count = _ok(cu.cuGraphGetEdges_v2(graph, count))
    before, overlapped = {}, {}
    for f, t, d in zip(froms, tos, data):
        assert int(t) not in before     # one stream: a chain
        before[int(t)] = int(f)
        if int(d.type) == int(cu.CUgraphDependencyType.CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC):
            overlapped[int(t)] = int(f)
    kernels = {}
    for n in nodes:
        if _ok(cu.cuGraphNodeGetType(n)) == cu.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            p = _ok(cu.cuGraphKernelNodeGetParams(n))
            kernels[int(n)] = (_ok(cu.cuFuncGetName(p.func)).decode(), p.gridDimX * p.gridDimY * p.gridDimZ, p.sharedMemBytes)
    after = {f: t for t, f in before.items()}
    order = [int(n) for n in nodes if int(n) not in before]
    while order and order[-1] in after:
        order.append(after[order[-1]])
    assert len(order) == len(nodes)
    made = [Launch(*kernels[n], kernels[overlapped[n]][0] if n in overlapped else None) for n in order if n in kernels]
    _ok(cu.cuGraphDestroy(graph))
    return made
