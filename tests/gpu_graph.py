"""The kernels a call launches, read from a CUDA graph it is captured into (nothing runs):
their names, the share of L1 they ask for as shared memory, the blocks of them an SM holds."""
import collections

Kernel = collections.namedtuple("Kernel", "name split block blocks_per_sm")


def _ok(result):
    error, *values = result
    assert int(error) == 0, error
    return values[0] if len(values) == 1 else values


def _kernels(driver, graph):
    _, count = _ok(driver.cuGraphGetNodes(graph, 0))
    nodes, _ = _ok(driver.cuGraphGetNodes(graph, count))
    types = driver.CUgraphNodeType
    split = driver.CUlaunchAttributeID.CU_LAUNCH_ATTRIBUTE_PREFERRED_SHARED_MEMORY_CARVEOUT
    found = []
    for node in nodes:
        kind = _ok(driver.cuGraphNodeGetType(node))
        if kind == types.CU_GRAPH_NODE_TYPE_GRAPH:
            found += _kernels(driver, _ok(driver.cuGraphChildGraphNodeGetGraph(node)))
        elif kind == types.CU_GRAPH_NODE_TYPE_KERNEL:
            params = _ok(driver.cuGraphKernelNodeGetParams(node))
            func = params.func if int(params.func) else _ok(driver.cuKernelGetFunction(params.kern))
            asked = _ok(driver.cuGraphKernelNodeGetAttribute(node, split)).sharedMemCarveout
            block = params.blockDimX * params.blockDimY * params.blockDimZ
            found.append(Kernel(
                _ok(driver.cuFuncGetName(func)).decode(), asked, block,
                _ok(driver.cuOccupancyMaxActiveBlocksPerMultiprocessor(
                    func, block, params.sharedMemBytes))))
    return found


def kernels_of(call):
    """The Kernel of every launch of call(stream), in no order."""
    import torch
    from cuda.bindings import driver

    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    handle = driver.CUstream(stream.cuda_stream)
    _ok(driver.cuStreamBeginCapture(
        handle, driver.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_THREAD_LOCAL))
    try:
        call(stream.cuda_stream)
    finally:
        graph = _ok(driver.cuStreamEndCapture(handle))
    try:
        return _kernels(driver, graph)
    finally:
        _ok(driver.cuGraphDestroy(graph))
