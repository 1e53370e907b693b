"""SiLU.mul over unpitched tensors (one long row), pitched rows (more than the grid has) and widths that are no multiple of 8."""
import pytest
import torch

from sparseflow_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 2056), (70000, 8), (257, 4104), (5, 100), (2, 2047), (9999, 72), (4099, 16)])
@pytest.mark.parametrize("pitched", [False, True])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_silu_mul_layouts(rows, cols, pitched, dtype):
    both = torch.randn(rows, 2 * cols, device="cuda").to(dtype)
    g, u = both.chunk(2, dim=1)
    if not pitched:
        g, u = g.contiguous(), u.contiguous()
    y = ops.silu_mul(g, u)
    ref = torch.nn.functional.silu(g.double()) * u.double()
    # one rounding to 16 bits (2^-9 bf16, 2^-12 f16) plus a few ulp of the fp32 exponential; subnormal f16 results: half a step
    rel, step = (2.0 ** -8, 0.0) if dtype == torch.bfloat16 else (2.0 ** -11, 2.0 ** -25)
    assert ((y.double() - ref).abs() <= rel * ref.abs() + step + 1e-30).all()


@pytest.mark.parametrize("cols", [8, 64, 256])
def test_pitched_narrow_rows_keep_the_threads_busy(cols):
    """Rows of a wider tensor cost what they move: twice the lines of an unpitched tensor in narrow rows, not one block a row."""
    def time_us(g, u):
        for _ in range(3):
            ops.silu_mul(g, u)
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        for _ in range(20):
            ops.silu_mul(g, u)
        b.record()
        torch.cuda.synchronize()
        return a.elapsed_time(b) * 50
    n = 1 << 25
    g, u = torch.randn(n // cols, 2 * cols, device="cuda").to(torch.bfloat16).chunk(2, dim=1)
    assert time_us(g, u) < 3 * time_us(g.contiguous(), u.contiguous())      # 3-20 times with one block per row
