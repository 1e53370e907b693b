"""Gate / up biases in the SiLU.mul epilogue of every kernel that has one, and the module that uses them."""
import pytest
import torch

from sparseflow_b200 import ops
from sparseflow_b200.nn import SparseFlowMLP

pytestmark = pytest.mark.gpu
DT = {"f16": torch.float16, "bf16": torch.bfloat16}


@pytest.fixture
def force():
    yield ops.force_token_tile
    ops.force_token_tile(0)


def _ref(x, wg, wu, bg, bu):
    gate, up = (x.float() @ ops.decompress_24(ops.compress_weight(w)).float().t() for w in (wg, wu))
    gate = gate if bg is None else gate + bg.float()
    up = up if bu is None else up + bu.float()
    return torch.nn.functional.silu(gate) * up


# decode slabs, single-CTA tiles, pair tiles of 256 and 512 rows, band tiles without and with split K; ragged rows
@pytest.mark.parametrize("v,M", [(8, 3), (8, 20), (32, 20), (64, 50), (128, 100), (192, 200), (1240, 300), (1256, 300), (5240, 300),
                                 (2208, 210), (6080, 77), (6304, 300), (7080, 77), (9160, 150)])
@pytest.mark.parametrize("which", ["both", "gate", "up"])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_every_epilogue(force, v, M, which, dt):
    I, K = 208, 1600
    g = torch.Generator(device="cuda").manual_seed(v + M)
    wg, wu = ((torch.randn(I, K, generator=g, device="cuda") * 0.02).to(DT[dt]) for _ in range(2))
    bg, bu = (torch.randn(I, generator=g, device="cuda").to(DT[dt]) for _ in range(2))
    bg, bu = bg if which != "up" else None, bu if which != "gate" else None
    x = torch.randn(M, K, generator=g, device="cuda").to(DT[dt])
    force(v)
    y = ops.sparse_gemm_swiglu(x, ops.compress_gate_up(wg, wu), gate_bias=bg, up_bias=bu).float()
    assert ops.device_status() == 0
    ref = _ref(x, wg, wu, bg, bu)
    floor = 1e-2 * ref.pow(2).mean().sqrt()
    assert ((y - ref).abs() / torch.maximum(ref.abs(), floor)).max() <= 1e-2      # one 16-bit rounding, as the other GEMM tests


def test_module_reads_its_biases_at_every_call():
    H, I, dt = 256, 704, torch.float16
    wg, wu = ((torch.randn(I, H, device="cuda") * 0.02).to(dt) for _ in range(2))
    wd = (torch.randn(H, I, device="cuda") * 0.02).to(dt)
    bg, bu = (torch.randn(I, device="cuda").to(dt) for _ in range(2))
    m = SparseFlowMLP(H, I, wg, wu, wd, gate_bias=bg, up_bias=bu)
    x = torch.randn(2, 24, H, device="cuda").to(dt)

    def check(bg, bu):
        h = _ref(x.view(48, H), wg, wu, bg, bu).to(dt)
        ref = h.float() @ wd.float().t()
        err = (m(x).view(48, H).float() - ref).norm() / ref.norm()
        assert err <= 1.5e-3      # gate, up, hidden and output rounded to 11 bits: a few times 2^-12
    check(bg, bu)
    m.gate_bias.mul_(2)
    m.up_bias.zero_()
    check(m.gate_bias, m.up_bias)
    with pytest.raises(ValueError):
        ops.sparse_gemm_swiglu(x.view(48, H), ops.compress_gate_up(wg[:192], wu[:192]), gate_bias=bg)
