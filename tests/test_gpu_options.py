"""Options that choose how kernels are launched, seen in captured graphs.  Needs a B200."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def programmatic_edges(torch, run):
    """Of the graph that captures `run`: how many dependencies are programmatic (the dependent starts early)."""
    run()
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        run()
    get = ctypes.CDLL("libcuda.so.1").cuGraphGetEdges_v2
    get.argtypes = [ctypes.c_void_p] * 5
    count = ctypes.c_size_t()
    assert get(graph.raw_cuda_graph(), None, None, None, ctypes.byref(count)) == 0
    n = count.value
    ends, data = (ctypes.c_void_p * n)(), (ctypes.c_uint8 * (8 * n))()  # CUgraphEdgeData: from port, to port, type, 5 reserved bytes
    assert get(graph.raw_cuda_graph(), ends, (ctypes.c_void_p * n)(), data, ctypes.byref(count)) == 0
    return sum(data[8 * i + 2] == 1 for i in range(n))  # CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC


@pytest.mark.parametrize("option,m", [("gemv_pdl", 2), ("gemm_pdl", 64)])
def test_programmatic_launches_can_be_switched_off(gk, option, m):
    """Two products behind one another, each a staging launch and the product: three early starts, none with the option at 0, and
    the same results.  A context that has launched a wait for another rank starts its products early, but not their staging."""
    import torch
    K = gk.GpuKernels(0)
    n, k = 256, 512
    qt = gk.QuantType.q6k()
    blocks = torch.randint(0, 256, (n * (k // 256), 210), dtype=torch.uint8, device="cuda")
    blocks[:, 208:210] = torch.full((blocks.shape[0],), 0.01, device="cuda", dtype=torch.float16).view(torch.uint8).view(-1, 2)
    w = K.upload(qt, n, k, blocks.reshape(-1))
    x, y = torch.randn((m, k), device="cuda"), torch.empty((m, n), device="cuda")
    product = (lambda: K.gemv(w, x, y=y)) if option == "gemv_pdl" else (lambda: K.gemm(w, x, y=y))

    def run():
        product()
        product()

    assert programmatic_edges(torch, run) == 3
    product()
    want = y.clone()
    K.set(option, 0)
    assert programmatic_edges(torch, run) == 0
    y.zero_()
    product()
    assert torch.equal(y, want)
    K.set(option, 1)
    flags = torch.zeros(64, dtype=torch.int32, device="cuda")
    flags[1] = 1  # the other rank has signalled already
    theirs = torch.zeros(64, dtype=torch.int32, device="cuda")
    K.peer_barrier(flags.data_ptr(), [theirs.data_ptr()], rank=0, seq=1)
    torch.cuda.synchronize()
    assert programmatic_edges(torch, run) == 2
    assert K.status() == 0
    K.close()
