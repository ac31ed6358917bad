"""``ops.launch_count()`` against the kernels that a capture of the same call holds."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _kernels(call):
    """(kernels counted, kernels captured) of ``call``."""
    from cuda.bindings import runtime
    from photon_infer_b200.kernels import ops
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    before = ops.launch_count()
    with torch.cuda.graph(graph):
        call()
    counted = ops.launch_count() - before
    raw = runtime.cudaGraph_t(init_value=graph.raw_cuda_graph())
    _, _, n = runtime.cudaGraphGetNodes(raw, 0)
    _, nodes, n = runtime.cudaGraphGetNodes(raw, n)
    kinds = [runtime.cudaGraphNodeGetType(node)[1] for node in nodes[:n]]
    return counted, sum(k == runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds)


@pytest.mark.parametrize("M,N,K", [(1, 2048, 2048), (9, 2048, 8192), (300, 16384, 2048), (4096 + 33, 2048, 2048)])
def test_32_bit_products(M, N, K):
    from photon_infer_b200.kernels import ops
    x, w, out = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV), torch.empty(M, N, device=DEV)
    assert ops.sgemm_tc_supported(w)
    counted, captured = _kernels(lambda: ops.linear(x, w, out))
    assert counted == captured


@pytest.mark.parametrize("mode", ["state_space", "matrix_memory", "decay_rows"])
@pytest.mark.parametrize("way", ["walk", "segments", "chunks"])
def test_recurrences(mode, way):
    from photon_infer_b200.kernels import ops
    if mode == "decay_rows" and way == "walk":
        pytest.skip("gated linear attention has a kernel of its own")
    H, N, dv, T = 4, 64, 64, 320
    rand = lambda *shape: torch.randn(*shape, device=DEV)
    i32 = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)
    q, k, v, gates, p = rand(T, H * N), rand(T, H * N), rand(T, H * dv), rand(T, 2 * H), rand(H)
    memory, rows = mode == "matrix_memory", mode == "decay_rows"
    a = torch.sigmoid(rand(T, H * N)) if rows else None
    ga, gb = (None if rows else gates[:, :H]), (gates[:, H:] if memory else None)
    p0, p1, p2 = (None if rows else p), (None if rows else p), (p if mode == "state_space" else None)
    state, out, cu, slots = rand(1, H * N * dv + H * N + H), rand(T, H * dv), i32([0, T]), i32([0])
    tail = (p0, p1, p2, 6.0 if memory else 0.0, 1.0, cu, slots, state, out)
    if way == "walk":
        call = lambda: ops.linrec(mode, q, k, v, ga, gb, *tail, 1, H, H, N, dv, None)
    elif way == "segments":
        call = lambda: ops.linrec_segments(mode, q, k, v, a, ga, gb, *tail, [T], H, H, N, dv, None, segment=64)
    else:
        call = lambda: ops.linrec_chunks(mode, q, k, v, a, ga, gb, *tail, [T], H, H, N, dv, None)
    counted, captured = _kernels(call)
    assert counted == captured
