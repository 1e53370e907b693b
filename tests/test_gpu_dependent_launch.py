"""Kernels launched as programmatic dependents: a chain whose links write what the next ones read, eagerly, from two streams and
as a captured graph behind other kernels."""
import ctypes as C

import pytest
import torch

from sparseflow_b200 import ops

pytestmark = pytest.mark.gpu


def _chain(x, ws, after=lambda t: t):
    """Compression, gate|up, down and SiLU.mul back to back, each on the previous one's output."""
    gu, down = after(ops.compress_gate_up(ws[0], ws[1])), after(ops.compress_weight(ws[2]))
    y = after(ops.sparse_gemm(after(ops.sparse_gemm_swiglu(x, gu)), down))
    y = after(ops.silu_mul(y, x))
    return after(ops.sparse_gemm(after(ops.sparse_gemm_swiglu(y, gu)), down))


def _one_at_a_time(t):
    torch.cuda.synchronize()
    return t


@pytest.mark.parametrize("M", [1, 20, 70, 300, 1500])
def test_chain_of_dependent_launches(M):
    H, I = 1024, 2816
    g = torch.Generator(device="cuda").manual_seed(M)
    ws = [(torch.randn(r, k, generator=g, device="cuda") * 0.02).to(torch.bfloat16) for r, k in ((I, H), (I, H), (H, I))]
    x = torch.randn(M, H, generator=g, device="cuda").to(torch.bfloat16)
    ref = _chain(x, ws, _one_at_a_time)
    for _ in range(20):
        assert torch.equal(_chain(x, ws), ref)
    streams, outs = [torch.cuda.Stream() for _ in range(2)], []
    for s in streams:
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            outs += [_chain(x, ws) for _ in range(5)]
    torch.cuda.synchronize()
    assert all(torch.equal(o, ref) for o in outs)

    xs, s = torch.empty_like(x), streams[0]
    with torch.cuda.stream(s):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            xs.zero_()
            xs.add_(x)
            out = _chain(xs, ws)
        for _ in range(3):
            graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref) and ops.device_status() == 0


class _Edge(C.Structure):
    _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]


def _dependent(run):
    """Whether the second of two captured launches may start before the first has completed (a programmatic edge, type 1)."""
    run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        run()
        run()
    ends, edges, n = (C.c_void_p * 8)(), (_Edge * 8)(), C.c_size_t(8)
    get = C.CDLL("libcudart.so.12").cudaGraphGetEdges_v2
    assert get(C.c_void_p(graph.raw_cuda_graph()), ends, (C.c_void_p * 8)(), edges, C.byref(n)) == 0 and n.value == 1
    return edges[0].type == 1


# (rows, K, tokens, dependent): a partial pass with few tokens and long K starts after its predecessor; a full pass, 16 tokens,
# short K and the other kernels overlap it
@pytest.mark.parametrize("N,K,M,dependent", [(10720, 5888, 6, False), (14208, 4096, 15, False), (14336, 4096, 6, True), (10720, 5888, 16, True),
                                             (10720, 3072, 6, True), (10720, 5888, 1, True), (4096, 4096, 20, True), (10720, 4096, 300, True)])
def test_which_launches_overlap_their_predecessor(N, K, M, dependent):
    cw = ops.compress_weight((torch.randn(N, K, device="cuda") * 0.02).to(torch.bfloat16))
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    out = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    assert _dependent(lambda: ops.sparse_gemm(x, cw, out=out)) == dependent
