"""Sparse GEMM on the GPU through the C ABI against the fp32 oracle on the same pruned weights.

Tolerance (stated by the benchmark definition): max relative error <= 1e-2 against the
fp32-accumulated reference, relative to max(|ref|, 1e-2 * rms(ref)); the reference's own absolute
bound for its 11 production shapes (< 0.2, tests/validate_sparseflow_production.py:43) is asserted
as well."""
import numpy as np
import pytest
import torch

import oracle as o
from sparseflow_b200 import ops
from tests.util import bits_of, seeded_act, seeded_weight, to_dev

pytestmark = pytest.mark.gpu
REL_TOL = 1e-2


@pytest.fixture(autouse=True)
def _auto_tile():
    ops.force_token_tile(0)
    yield
    ops.force_token_tile(0)


def _run(R, K, M, dt, bn=0, sigma=0.02, wseed=1, xseed=1234, bias=False, act=None):
    w = seeded_weight(R, K, dt, wseed, sigma)
    x = seeded_act(M, K, dt, xseed)
    oc = o.prune_24(w, dt)
    cw = ops.compress_weight(to_dev(w, dt))
    ref = o.gemm_ref(x, oc["pruned"], dt)
    bt = None
    if bias:
        b = seeded_act(1, R, dt, 77)[0]
        bt = to_dev(b, dt)
        ref = ref + o.to_f32(b, dt)[None, :]
    if act == "relu":
        ref = np.maximum(ref, 0)
    elif act == "silu":
        ref = ref / (1 + np.exp(-ref))
    elif act == "gelu":
        ref = torch.nn.functional.gelu(torch.from_numpy(ref)).numpy()
    ops.force_token_tile(bn)
    y = ops.sparse_gemm(to_dev(x, dt), cw, bias=bt, act=act)
    assert ops.device_status() == 0
    return o.to_f32(bits_of(y), dt), ref


@pytest.mark.parametrize("bn,R,K,M", [(64, 128, 64, 64), (128, 128, 128, 128), (256, 128, 256, 256),
                                      (1256, 256, 256, 256), (1240, 512, 256, 240), (1192, 256, 192, 192),
                                      (2208, 512, 256, 208), (2240, 1024, 192, 240), (5240, 1024, 256, 240)])
def test_identity_activations_reproduce_pruned_weight_exactly(bn, R, K, M):
    dt = "bf16"
    w = seeded_weight(R, K, dt, 3)
    cw = ops.compress_weight(to_dev(w, dt))
    x = o.from_f32(np.eye(M, K, dtype=np.float32), dt)
    ops.force_token_tile(bn)
    y = ops.sparse_gemm(to_dev(x, dt), cw)
    assert ops.device_status() == 0
    n = min(K, M)
    assert (bits_of(y)[:n].T == o.prune_24(w, dt)["pruned"][:, :n]).all()


@pytest.mark.parametrize("bn", [32, 64, 128, 192, 256, 1256, 1240, 1224, 1208, 1192, 2192, 2208, 2224, 2240, 5240, 5224, 5208, 5192])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_every_kernel_variant_ragged(bn, dt):
    y, ref = _run(392, 512, 300, dt, bn=bn)
    assert o.rel_err_metrics(y, ref)["floor"] <= REL_TOL


@pytest.mark.parametrize("bn", [1240, 1224, 1208, 1192, 5240, 5192, 2240])
def test_two_accumulator_pair_tiles_many_tiles_per_pair(bn):
    """The 256-row tiles with two accumulator sets, on a problem with more tiles than SM pairs (5 row tiles
    x 9-11 token tiles on 74 pairs would be one tile each; 24 row tiles x 9-11 gives every pair 3-4 tiles), so
    both accumulator sets and their phase bits are reused; bias + activation in the epilogue."""
    y, ref = _run(6144 - 8, 256, 2000, "bf16", bn=bn, bias=True, act="relu")
    assert o.rel_err_metrics(y, ref)["floor"] <= REL_TOL


@pytest.mark.parametrize("M", [1, 8, 33, 77, 128, 1000])
def test_ragged_token_counts_auto_dispatch(M):
    y, ref = _run(1000, 1024, M, "bf16")
    assert y.shape == (M, 1000)
    assert o.rel_err_metrics(y, ref)["floor"] <= REL_TOL


@pytest.mark.parametrize("M", [1, 5, 8, 9, 16, 24, 32])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_small_m_kernel(M, dt):
    """Decode kernel (warp-level mma.sp), forced for every M it supports; K with a 64-wide tail."""
    y, ref = _run(1000, 1024 + 64, M, dt, bn=8, bias=True)
    assert y.shape == (M, 1000)
    assert o.rel_err_metrics(y, ref)["floor"] <= REL_TOL


def test_small_m_kernel_mistral_down_shape():
    y, ref = _run(4096, 14336, 8, "bf16", bn=8)
    assert o.rel_err_metrics(y, ref)["floor"] <= REL_TOL


@pytest.mark.parametrize("bn", [128, 1256, 1240, 2208, 5240])
@pytest.mark.parametrize("act", [None, "relu", "silu", "gelu"])
def test_bias_and_activation_epilogues(bn, act):
    y, ref = _run(256, 512, 200, "f16", bn=bn, bias=True, act=act)
    assert o.rel_err_metrics(y, ref)["floor"] <= REL_TOL


# ---- split-K over a cluster (3000 + token tile = 2 K-slices, 4000 + token tile = 4 K-slices)
@pytest.mark.parametrize("bn,M", [(3032, 20), (3064, 40), (3128, 100), (4032, 32), (4064, 64), (4128, 128),
                                  (4128, 300)])
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_split_k_variants_ragged(bn, M, dt):
    """Rows not a multiple of 128, K with a 64-wide tail (9 metadata tiles split 3/2/2/2), ragged tokens."""
    y, ref = _run(392, 1024 + 64, M, dt, bn=bn)
    assert y.shape == (M, 392)
    assert o.rel_err_metrics(y, ref)["floor"] <= REL_TOL


@pytest.mark.parametrize("bn", [3064, 4128])
def test_split_k_identity_is_exact(bn):
    dt, R, K, M = "bf16", 256, 1024, 128
    w = seeded_weight(R, K, dt, 3)
    cw = ops.compress_weight(to_dev(w, dt))
    x = o.from_f32(np.eye(M, K, dtype=np.float32), dt)
    ops.force_token_tile(bn)
    y = ops.sparse_gemm(to_dev(x, dt), cw)
    assert ops.device_status() == 0
    assert (bits_of(y).T == o.prune_24(w, dt)["pruned"][:, :M]).all()


@pytest.mark.parametrize("act", [None, "relu", "silu", "gelu"])
def test_split_k_bias_and_activation(act):
    y, ref = _run(256, 2048, 96, "f16", bn=4128, bias=True, act=act)
    assert o.rel_err_metrics(y, ref)["floor"] <= REL_TOL


@pytest.mark.parametrize("R,K,M", [(4096, 11008, 16), (4096, 11008, 128), (4096, 4096, 64), (4096, 14336, 256),
                                   (8192, 8192, 32)])
def test_split_k_auto_dispatch_on_few_row_tiles(R, K, M):
    """Shapes the dispatcher sends to the split-K kernel (32 or 64 row tiles on 148 SMs); the result is
    also bit-identical from one launch to the next (fixed summation order, no atomics)."""
    dt = "bf16"
    w = seeded_weight(R, K, dt, 6)
    x = seeded_act(M, K, dt, 7)
    cw = ops.compress_weight(to_dev(w, dt))
    xd = to_dev(x, dt)
    y1 = ops.sparse_gemm(xd, cw)
    y2 = ops.sparse_gemm(xd, cw)
    assert ops.device_status() == 0
    assert torch.equal(y1, y2)
    ref = o.gemm_ref(x, o.prune_24_pruned_chunked(w, dt), dt)
    assert o.rel_err_metrics(o.to_f32(bits_of(y1), dt), ref)["floor"] <= REL_TOL


@pytest.mark.parametrize("bn", [0, 1240, 2240, 5240])
def test_pair_kernel_l2_band_tile_order(bn):
    """Enough token tiles at K = 8192 that the prefill kernel walks them in more than one L2 band
    (12-13 token tiles, bands of 6-7), with ragged rows and tokens."""
    y, ref = _run(520, 8192, 3000, "bf16", bn=bn)
    assert y.shape == (3000, 520)
    assert o.rel_err_metrics(y, ref)["floor"] <= REL_TOL


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("bn", [1256, 1240, 5240])
def test_pair_kernel_both_tile_orders_many_bands(order, bn):
    """Either operand as the L2-resident one (bands of token tiles / bands of row tiles), with the band budget
    turned down to 1 MB so that a small problem walks several bands of each kind: 5 row tiles (3 at 512 rows) and
    9-10 token tiles at K = 2048, ragged in rows and tokens."""
    from sparseflow_b200 import _lib
    L = _lib.lib()
    try:
        assert L.sfb200_debug_pair_tuning(1, order) == 0
        y, ref = _run(1160, 2048, 2300, "bf16", bn=bn, bias=True)
    finally:
        assert L.sfb200_debug_pair_tuning(40, -1) == 0
    assert y.shape == (2300, 1160)
    assert o.rel_err_metrics(y, ref)["floor"] <= REL_TOL


@pytest.mark.parametrize("bn", [0, 1256, 1240, 5240])
@pytest.mark.parametrize("M", [40, 1000])
def test_fp32_output_epilogue(bn, M):
    """sfb200_sparse_gemm_f32out: the fp32 accumulators (+ bias) stored unrounded, for partial sums that are added
    before they are rounded.  Against the fp32 oracle the only difference left is summation order."""
    from sparseflow_b200 import _lib
    dt, R, K = "bf16", 1160, 1024 + 64
    w, x = seeded_weight(R, K, dt, 8), seeded_act(M, K, dt, 9)
    b = seeded_act(1, R, dt, 10)[0]
    cw = ops.compress_weight(to_dev(w, dt))
    xd, bd = to_dev(x, dt), to_dev(b, dt)
    y = torch.full((M, R), float("nan"), device="cuda", dtype=torch.float32)
    ops.force_token_tile(bn)
    rc = _lib.lib().sfb200_sparse_gemm_f32out(xd.data_ptr(), K, cw.values.data_ptr(), cw.meta.data_ptr(), y.data_ptr(), R,
                                              M, R, K, ops.BF16, bd.data_ptr(), 0, torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and ops.device_status() == 0
    ref = o.gemm_ref(x, o.prune_24(w, dt)["pruned"], dt) + o.to_f32(b, dt)[None, :]
    got = y.cpu().numpy()
    assert np.isfinite(got).all()
    m = o.rel_err_metrics(got, ref)
    assert m["chain"] <= 1e-5 and m["floor"] <= 1e-3, m      # relative to the rms / to max(|ref|, 1e-2 rms)


@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("bn,rank", [(0, 0), (1240, 2), (5240, 1), (1256, 3)])
def test_scatter_epilogue_slot_kinds_on_one_gpu(kind, bn, rank):
    """sfb200_sparse_gemm_scatter with the four "owners'" receive slots in THIS GPU's memory (stores only, nothing waits):
    token block o of the product lands in slot o, as the weight dtype (kind 0), float (1) or clamped fp16 (2), whatever
    block the rank starts its token tiles at.  Rows of a slot beyond the block's live tokens stay untouched."""
    import ctypes as C
    from sparseflow_b200 import _lib
    from sparseflow_b200.parallel import block_rows
    dt, R, K, M, tp = "bf16", 1160, 1024 + 64, 1000, 4
    w, x = seeded_weight(R, K, dt, 21), seeded_act(M, K, dt, 22)
    cw = ops.compress_weight(to_dev(w, dt))
    xd = to_dev(x, dt)
    mo = block_rows(M, tp)
    tdt = {0: torch.bfloat16, 1: torch.float32, 2: torch.float16}[kind]
    slots = torch.full((tp, mo, R), 7.0, device="cuda", dtype=tdt)
    ptrs = (C.c_void_p * 8)(*[slots[o].data_ptr() if o < tp else None for o in range(8)])
    ops.force_token_tile(bn)
    rc = _lib.lib().sfb200_sparse_gemm_scatter(xd.data_ptr(), K, cw.values.data_ptr(), cw.meta.data_ptr(),
                                               C.cast(ptrs, C.POINTER(C.c_void_p)), tp, rank, mo, kind, M, R, K, ops.BF16,
                                               torch.cuda.current_stream().cuda_stream)
    ops.force_token_tile(0)
    assert rc == 0 and ops.device_status() == 0
    ref = o.gemm_ref(x, o.prune_24(w, dt)["pruned"], dt)
    got = slots.float().cpu().numpy().reshape(tp * mo, R)
    m = o.rel_err_metrics(got[:M], ref)
    assert m["floor"] <= (1e-3 if kind == 1 else REL_TOL), m
    assert (got[M:] == 7.0).all()          # the dead rows of the last owner's slot


def test_config1_fp16_m512_k4096_n4096():
    y, ref = _run(4096, 4096, 512, "f16", wseed=1, xseed=1234)
    m = o.rel_err_metrics(y, ref)
    assert m["floor"] <= REL_TOL and m["norm"] <= REL_TOL, m
    # must-fail sanity check (tests/validate_correctness_REAL.py:74-78): a corrupted output is caught
    bad = y.copy()
    bad.reshape(-1)[0] += 1.0
    assert o.rel_err_metrics(bad, ref)["floor"] > REL_TOL


PRODUCTION_SHAPES = [   # (sparse rows, dense cols, K) of tests/validate_sparseflow_production.py:47-59
    (512, 512, 512), (1024, 1024, 1024), (2048, 2048, 2048), (4096, 4096, 4096),
    (128, 4096, 4096), (512, 4096, 4096), (2048, 4096, 4096),
    (512, 11008, 4096), (2048, 11008, 4096), (512, 4096, 11008), (2048, 4096, 11008),
]


@pytest.mark.parametrize("R,T,K", PRODUCTION_SHAPES)
def test_reference_production_shapes_fp16_unit_normal(R, T, K):
    """Both operands N(0,1) fp16, seed 42, as the reference validates; abs error < 0.2."""
    y, ref = _run(R, K, T, "f16", sigma=1.0, wseed=42, xseed=43)
    m = o.rel_err_metrics(y, ref)
    # reference bound: < 0.2 absolute.  fp16 cannot do better than half an ulp of the largest output
    # (0.25 once |y| >= 512, which the K = 11008 shapes reach), so the bound is widened to that.
    assert m["max_abs"] < max(0.2, float(np.abs(ref).max()) * 2.0 ** -10), m
    assert m["floor"] <= REL_TOL, m


@pytest.mark.parametrize("bn", [0, 192])
def test_full_size_identity_property_llama_gate_up(bn):
    """Size-independent exact check at the benchmark's full weight size: with one-hot activations
    the GEMM must return the pruned weight itself (22016 x 4096, M = 4096 tokens)."""
    dt = "bf16"
    g = torch.Generator(device="cuda").manual_seed(5)
    w = (torch.randn(22016, 4096, generator=g, device="cuda", dtype=torch.float32) * 0.02).to(torch.bfloat16)
    cw = ops.compress_weight(w)
    x = torch.eye(4096, device="cuda", dtype=torch.bfloat16)
    ops.force_token_tile(bn)
    y = ops.sparse_gemm(x, cw)
    assert ops.device_status() == 0
    assert torch.equal(y.t().contiguous(), ops.decompress_24(cw))


def test_argument_errors_are_reported():
    w = to_dev(seeded_weight(128, 128, "bf16", 1), "bf16")
    cw = ops.compress_weight(w)
    with pytest.raises(ValueError):
        ops.sparse_gemm(torch.zeros(4, 64, device="cuda", dtype=torch.bfloat16), cw)       # wrong K
    with pytest.raises(ValueError):
        ops.sparse_gemm(torch.zeros(4, 128, device="cuda", dtype=torch.float16), cw)       # dtype mismatch
    with pytest.raises(ValueError):
        ops.sparse_gemm(torch.zeros(4, 128, dtype=torch.bfloat16), cw)                      # not CUDA
    w2 = to_dev(seeded_weight(128, 96, "bf16", 1), "bf16")                                  # K % 64 != 0
    cw2 = ops.compress_weight(w2)
    from sparseflow_b200._lib import SfbError
    with pytest.raises(SfbError):
        ops.sparse_gemm(torch.zeros(4, 96, device="cuda", dtype=torch.bfloat16), cw2)


def test_random_shapes_through_the_dispatcher():
    """Seeded random (tokens, rows, K) triples, ragged in every dimension the library allows (rows % 8 == 0,
    K % 64 == 0), through whatever kernel the dispatcher picks, against an fp32 matmul on the decompressed
    weight (GPU reference: the decompression itself is pinned bit-exactly elsewhere)."""
    from sparseflow_b200 import _lib
    rng = np.random.default_rng(2024)
    seen = set()
    for case in range(48):
        M = int(rng.choice([1, 2, 3, 5, 8, 9, 17, 31, 33, 64, 65, 100, 129, 200, 257, 384, 513, 700, 1023, 1024, 1500]))
        N = int(rng.choice([8, 24, 120, 128, 136, 392, 512, 1000, 2048, 4096, 4104]))
        K = int(rng.choice([64, 128, 192, 576, 1024, 1088, 2048, 4160]))
        seen.add(_lib.lib().sfb200_debug_plan_gemm(M, N, K, 0, 148))
        g = torch.Generator(device="cuda").manual_seed(case)
        w = (torch.randn(N, K, generator=g, device="cuda") * 0.05).to(torch.bfloat16)
        x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
        cw = ops.compress_weight(w)
        y = ops.sparse_gemm(x, cw).float()
        ref = x.float() @ ops.decompress_24(cw).float().t()
        floor = 1e-2 * ref.pow(2).mean().sqrt()
        rel = ((y - ref).abs() / torch.maximum(ref.abs(), floor)).max().item()
        assert y.shape == (M, N) and rel <= REL_TOL, (M, N, K, rel)
    assert ops.device_status() == 0
    # decode, single-CTA tiles, split-K, pair tiles, band tiles without and with split K were all exercised
    families = {"decode" if v == 8 else "single" if v < 1000 else "pair" if v < 3000 or 5000 <= v < 6000 else
                "split K" if v < 5000 else "band" if v < 7000 else "band, split K" for v in seen}
    assert len(families) == 6, seen


# both sides of every token count at which the dispatcher changes its candidates
@pytest.mark.parametrize("M", [1, 4, 5, 8, 9, 32, 33, 64, 65, 128, 129, 160, 161, 800, 801, 1023, 1024])
@pytest.mark.parametrize("N,K,swiglu", [(392, 1088, 0), (2048, 2048, 0), (4736, 1024, 0), (8704, 1216, 0), (416, 1088, 1), (8192, 1024, 1)])
def test_dispatch_boundaries(M, N, K, swiglu):
    """Nothing forced: whatever the dispatcher picks, in both epilogues, against an fp32 matmul on the decompressed weight."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    ws = [(torch.randn(N // (1 + swiglu), K, generator=g, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(1 + swiglu)]
    cws = [ops.compress_weight(w) for w in ws]
    y = (ops.sparse_gemm_swiglu(x, ops.compress_gate_up(*ws)) if swiglu else ops.sparse_gemm(x, cws[0])).float()
    assert ops.device_status() == 0
    refs = [x.float() @ ops.decompress_24(cw).float().t() for cw in cws]
    ref = torch.nn.functional.silu(refs[0]) * refs[1] if swiglu else refs[0]
    floor = 1e-2 * ref.pow(2).mean().sqrt()
    assert ((y - ref).abs() / torch.maximum(ref.abs(), floor)).max().item() <= REL_TOL
