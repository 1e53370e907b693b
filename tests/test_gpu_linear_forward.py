"""``SparseFlowLinear.forward`` on both branches: call counters, no autograd graph, leading shapes."""
import pytest
import torch

from sparseflow_b200.nn import SparseFlowLinear, SparseFlowPolicy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 128), (2, 3, 128), (0, 128), (128,)])
@pytest.mark.parametrize("sparse", [True, False])
def test_forward_counts_and_builds_no_graph(shape, sparse):
    w = (torch.randn(64, 128, device="cuda") * 0.02).to(torch.float16)
    policy = SparseFlowPolicy(decode_max_M_o=1 << 20) if sparse else SparseFlowPolicy(decode_max_M_o=0, min_M_o=1 << 20)
    m = SparseFlowLinear(w, None, policy=policy, op_name="o_proj", dense_uses_pruned=True)
    x = torch.randn(shape, device="cuda").to(torch.float16).requires_grad_()
    y = m(x)
    empty = x.numel() == 0                    # an empty batch is never sparse
    assert (m._sparse_count, m._dense_count) == ((1, 0) if sparse and not empty else (0, 1))
    assert y.shape == (*shape[:-1], 64) and not y.requires_grad and y.grad_fn is None
    ref = x.detach().float() @ m.W_dense_pruned.float().t()
    assert torch.allclose(y.float(), ref, rtol=2e-3, atol=2e-3)      # one fp16 rounding (2^-11) and fp32 summation order
