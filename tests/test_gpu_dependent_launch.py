"""Kernels launched as programmatic dependents: a chain whose links write what the next ones read, eagerly, from two streams and
as a captured graph behind other kernels."""
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
