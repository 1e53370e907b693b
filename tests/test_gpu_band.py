"""CTA-pair GEMM for token counts between decode and prefill (force 6000 / 7000 / 9000 / 8000 + token tile = K split over 1 / 2 / 3 / 4
pairs), against an fp32 matmul on the decompressed weight and against a fixed-tile kernel on the same call."""
import pytest
import torch

from sparseflow_b200 import _lib, ops

REL_TOL = 1e-2        # one 16-bit rounding, relative to max(|ref|, 1e-2 rms): the bound of the other GEMM tests
DT = {"f16": torch.float16, "bf16": torch.bfloat16}


def test_band_forms_have_legal_tiles():
    """Band forms only from 33 to 1023 tokens, with a tile of 16 to 400 tokens and at least 512 of K per slice; both planning
    calls give the same answer."""
    plan, route = _lib.lib().sfb200_debug_plan_gemm, _lib.lib().sfb200_debug_route_gemm
    for sms in (148, 132, 64, 2):
        for N, K in ((4096, 4096), (22016, 4096), (4096, 11008), (57344, 8192), (8, 64), (392, 1088), (1024, 512)):
            for M in (1, 2, 5, 8, 32, 33, 64, 65, 100, 160, 161, 256, 257, 300, 512, 777, 1023, 1024, 5000):
                v = plan(M, N, K, 0, sms)
                assert v == route(M, N, K, 0, sms)
                if v >= 6000:
                    t = v % 1000
                    assert 32 < M < 1024 and v < 10000 and 16 <= t <= 400 and t % 16 == 0, (M, N, K, sms, v)
                    assert v < 7000 or K > 512 * {7: 2, 9: 3, 8: 4}[v // 1000] - 128, (M, N, K, sms, v)
    assert plan(0, 8, 64, 0, 148) == 0 and route(0, 8, 64, 0, 148) == 0


@pytest.fixture
def force():
    yield ops.force_token_tile
    ops.force_token_tile(0)


def _close(y, ref):
    floor = 1e-2 * ref.pow(2).mean().sqrt()
    return ((y.float() - ref).abs() / torch.maximum(ref.abs(), floor)).max().item() <= REL_TOL


# (M, N, K, variant): one tile; rows below a tile; K with a 64-wide tail; uneven K slices; a ragged last token block;
# several passes with both accumulator sets; left-over tiles cut into slices (172 = 148 + 24 tiles, 3 slices; 86 = 74 + 12,
# 6 slices, the last one empty of tokens); tiles above 256 tokens (two MMAs of unequal width, slices in columns of their own,
# several K steps of a slice per ring stage with a remainder, the largest exchange); one accumulator set over several passes
CASES = [(64, 256, 256, 6064), (16, 8, 64, 6016), (300, 392, 1088, 6160), (300, 392, 1088, 7160), (300, 392, 1088, 8160),
         (300, 392, 1088, 9160), (77, 1160, 2048, 9080), (777, 520, 2048, 9400), (400, 22016, 640, 6208), (512, 28672, 256, 6256),
         (300, 22016, 256, 6304), (777, 11008, 384, 6400), (270, 256, 1088, 7272), (777, 520, 2048, 7400), (600, 392, 1088, 8304),
         (350, 264, 192, 6352), (1200, 20000, 128, 6400), (33, 1160, 2048, 8048), (500, 520, 2048, 7256), (2000, 6136, 256, 6240), (300, 22016, 256, 6160),
         (150, 22016, 256, 6160), (1, 264, 1024, 7016), (700, 20000, 128, 6256)]


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,v", CASES)
@pytest.mark.parametrize("dt,bias,act", [("bf16", False, None), ("f16", True, "gelu")])
def test_band_kernel_edges(force, M, N, K, v, dt, bias, act):
    """Strided activations and output, bias and activation; the padding of the output stays untouched."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    w = (torch.randn(N, K, generator=g, device="cuda") * 0.05).to(DT[dt])
    x = torch.randn(M, K + 64, generator=g, device="cuda").to(DT[dt])[:, :K]
    b = torch.randn(N, generator=g, device="cuda").to(DT[dt]) if bias else None
    cw = ops.compress_weight(w)
    out = torch.full((M + 1, N + 8), 7.0, device="cuda", dtype=DT[dt])
    force(v)
    y = ops.sparse_gemm(x, cw, bias=b, act=act, out=out[:M, :N])
    y2 = ops.sparse_gemm(x, cw, bias=b, act=act)
    force(1240)
    fixed = ops.sparse_gemm(x, cw, bias=b, act=act)
    assert ops.device_status() == 0
    ref = x.float() @ ops.decompress_24(cw).float().t()
    ref = ref + b.float() if bias else ref
    ref = torch.nn.functional.gelu(ref) if act else ref
    assert _close(y, ref) and _close(fixed, ref)
    assert torch.equal(y, y2)                                  # fixed summation order
    assert (out[M] == 7.0).all() and (out[:, N:] == 7.0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("M,I,K,v", [(150, 11008, 256, 6160), (77, 208, 1088, 7080), (300, 48, 1024, 8160), (1000, 6000, 192, 6256)])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_band_kernel_swiglu(force, M, I, K, v, dt):
    g = torch.Generator(device="cuda").manual_seed(M + I)
    wg, wu = ((torch.randn(I, K, generator=g, device="cuda") * 0.05).to(DT[dt]) for _ in range(2))
    x = torch.randn(M, K, generator=g, device="cuda").to(DT[dt])
    cw = ops.compress_gate_up(wg, wu)
    force(v)
    y = ops.sparse_gemm_swiglu(x, cw)
    assert ops.device_status() == 0
    gate, up = (x.float() @ ops.decompress_24(ops.compress_weight(w)).float().t() for w in (wg, wu))
    assert _close(y, torch.nn.functional.silu(gate) * up)


@pytest.mark.gpu
@pytest.mark.parametrize("v", [6128, 7128, 8128, 9128, 9336])
def test_band_kernel_identity_is_exact(force, v):
    """One-hot activations return the pruned weight bit for bit, whichever pair owns a chunk."""
    w = (torch.randn(4096, 1024, device="cuda") * 0.02).to(torch.bfloat16)
    cw = ops.compress_weight(w)
    force(v)
    y = ops.sparse_gemm(torch.eye(1024, device="cuda", dtype=torch.bfloat16), cw)
    assert ops.device_status() == 0 and torch.equal(y.t().contiguous(), ops.decompress_24(cw))
