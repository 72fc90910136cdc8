"""What a call launches, read from a CUDA graph that it is captured into."""

import collections

import torch
from cuda.bindings import driver

Launch = collections.namedtuple("Launch", "name grid cluster")   # mangled name, CTAs, CTAs of a cluster


def _ok(result):
    assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
    return result[1] if len(result) == 2 else result[1:]


def launched(call):
    """The kernels of `call`, as a list of Launch. The call runs once before, on the same stream."""
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        call()
    raw = driver.CUgraph(graph.raw_cuda_graph())
    count = _ok(driver.cuGraphGetNodes(raw))[1]
    found = []
    for node in _ok(driver.cuGraphGetNodes(raw, count))[0][:count]:
        if _ok(driver.cuGraphNodeGetType(node)) != driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        params = _ok(driver.cuGraphKernelNodeGetParams(node))
        name = _ok(driver.cuFuncGetName(params.func)) if int(params.func) else _ok(driver.cuKernelGetName(params.kern))
        cluster = _ok(driver.cuGraphKernelNodeGetAttribute(node, driver.CUkernelNodeAttrID.CU_LAUNCH_ATTRIBUTE_CLUSTER_DIMENSION))
        found.append(Launch(name.decode(), params.gridDimX * params.gridDimY * params.gridDimZ, max(1, cluster.clusterDim.x)))
    return found
