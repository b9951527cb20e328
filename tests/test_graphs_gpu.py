"""FAST factors captured in CUDA graphs, looked at through the driver's own calls."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

MEM_ALLOC, MEM_FREE = 10, 11  # CU_GRAPH_NODE_TYPE_MEM_ALLOC, .._MEM_FREE


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_a_captured_factor_is_an_ordinary_graph(gpu_lla, dtype, mode):
    """In every capture mode: no allocation nodes; the graph can be cloned, instantiated twice and
    be a child of another, each instance gives the factor, and its scratch outlives the graph."""
    import torch
    cu = ctypes.CDLL("libcuda.so.1")

    def ok(code):
        assert code == 0, code

    n = 300
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    G = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    A = (G @ G.T / n + torch.eye(n, dtype=torch.float64, device="cuda")).to(getattr(torch, dtype))
    A = torch.tril(A) + torch.tril(A, -1).T
    L = A.clone().T
    info = gpu_lla.potrf_device(L, algo=gpu_lla.ALGO_FAST)
    torch.cuda.synchronize()
    want = L.clone()
    stream = torch.cuda.Stream()
    st = ctypes.c_void_p(stream.cuda_stream)
    graph, clone, parent, child = (ctypes.c_void_p() for _ in range(4))
    ok(cu.cuStreamBeginCapture_v2(st, mode))
    gpu_lla.potrf_device(L, algo=gpu_lla.ALGO_FAST, info=info, stream=stream)
    ok(cu.cuStreamEndCapture(st, ctypes.byref(graph)))
    count = ctypes.c_size_t()
    ok(cu.cuGraphGetNodes(graph, None, ctypes.byref(count)))
    nodes = (ctypes.c_void_p * count.value)()
    ok(cu.cuGraphGetNodes(graph, nodes, ctypes.byref(count)))
    for nd in nodes:
        kind = ctypes.c_int()
        ok(cu.cuGraphNodeGetType(ctypes.c_void_p(nd), ctypes.byref(kind)))
        assert kind.value not in (MEM_ALLOC, MEM_FREE)
    ok(cu.cuGraphClone(ctypes.byref(clone), graph))
    ok(cu.cuGraphCreate(ctypes.byref(parent), 0))
    ok(cu.cuGraphAddChildGraphNode(ctypes.byref(child), parent, None, ctypes.c_size_t(0), graph))
    execs = []
    for gr in (graph, graph, clone, parent):
        e = ctypes.c_void_p()
        ok(cu.cuGraphInstantiateWithFlags(ctypes.byref(e), gr, ctypes.c_ulonglong(0)))
        execs.append(e)
    for gr in (graph, clone, parent):
        ok(cu.cuGraphDestroy(gr))
    other = A.clone().T
    for e in execs:
        L.copy_(A.T)
        info.fill_(7)
        torch.cuda.synchronize()
        ok(cu.cuGraphLaunch(e, st))
        gpu_lla.potrf_device(other, algo=gpu_lla.ALGO_FAST)  # a call with scratch of its own beside it
        torch.cuda.synchronize()
        assert int(info.item()) == -1 and bool((L == want).all())
        other.copy_(A.T)
    for e in execs:
        ok(cu.cuGraphExecDestroy(e))
    gpu_lla.potrf_device(other, algo=gpu_lla.ALGO_FAST)
    torch.cuda.synchronize()
    assert bool((other == want).all())
