"""One-pass checked compression into a container against the separate check, compression and packing."""
import pytest
import torch

from sparseflow_b200 import _lib, core, ops, serialize

pytestmark = pytest.mark.gpu


def _special(shape, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = (torch.randn(shape, generator=g, device="cuda") * 0.02).to(dtype)
    n = max(2, w.numel() // 50)
    for v in (0.0, -0.0, float("inf"), float("nan"), w.flatten()[0].item()):
        w.view(-1)[torch.randint(0, w.numel(), (n,), generator=g, device="cuda")] = v
    return w


@pytest.mark.parametrize("rows,K", [(1, 16), (16, 48), (100, 64), (130, 528), (8, 4096), (1000, 1040)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_blob_equals_pack(rows, K, dtype):
    w = core.prune_2_4(_special((rows, K), dtype, rows + K))
    blob, valid = serialize.compress_checked(w)
    assert valid and torch.equal(blob, serialize.pack(ops.compress_weight(w)))
    assert torch.equal(core.compress_2_4(w), blob)
    wide = torch.empty(rows, K + 8, device="cuda", dtype=dtype)      # a row pitch of its own
    wide[:, :K] = w
    assert torch.equal(serialize.compress_checked(wide[:, :K])[0], blob)
    assert torch.equal(serialize.compress_checked(w.t().contiguous().t())[0], blob)
    assert ops.device_status() == 0


@pytest.mark.parametrize("where", [(0, 0), (129, 1036), (64, 512), (8, 3)])
def test_one_bad_group_is_found(where):
    w = torch.zeros(130, 1040, device="cuda", dtype=torch.float16)
    w.view(-1, 4)[:, 1:3] = 1.0
    assert serialize.compress_checked(w)[1]
    r, c = where
    w[r, c // 4 * 4] = -6e-8                                          # a third non-zero, the smallest subnormal
    assert not serialize.compress_checked(w)[1]
    with pytest.raises(ValueError):
        core.compress_2_4(w)


def test_forms_outside_the_one_pass_kernel_answer_as_before():
    """The same error as the separate check and compression, or the verdict of the check."""
    w = torch.zeros(32, 20, device="cuda", dtype=torch.float16)      # K % 16 != 0: no packed form
    odd = torch.zeros(33 * 64 + 1, device="cuda", dtype=torch.float16)[1:].view(33, 64)   # unaligned
    for t, step in ((w, ops.compress_weight), (odd, ops.validate_24)):
        with pytest.raises(_lib.SfbError) as alone:
            step(t)
        with pytest.raises(_lib.SfbError) as checked:
            core.compress_2_4(t)
        assert str(checked.value) == str(alone.value)
    dense = torch.ones(32, 20, device="cuda", dtype=torch.float16)   # not 2:4: found before the width is
    with pytest.raises(ValueError, match="2:4"):
        core.compress_2_4(dense)
    with pytest.raises(ValueError):
        core.compress_2_4(torch.zeros(32, 64, dtype=torch.float16))  # not on the GPU


@pytest.mark.parametrize("rows,K", [(1, 4), (3, 20), (37, 100), (64, 16), (129, 1012), (513, 4092)])
@pytest.mark.parametrize("tie", ["high", "low"])
def test_widths_that_are_multiples_of_four(rows, K, tie):
    """One run of elements (no row padding) against the group-by-group kernel, which a row pitch of its own selects."""
    w = _special((rows, K), torch.float16, K)
    wide = torch.empty(rows, K + 4, device="cuda", dtype=torch.float16)
    wide[:, :K] = w
    kw = dict(tie=tie, want_meta=False, want_ref_codes=True, want_pruned=True)
    flat, pitched = ops.prune_compress_24(w, **kw), ops.prune_compress_24(wide[:, :K], **kw)
    for name, t in pitched.items():
        assert torch.equal(flat[name].view(torch.uint8), t.view(torch.uint8)), name
    for m in (flat["pruned"], w):
        padded = torch.zeros(rows, K + 4, device="cuda", dtype=torch.float16)
        padded[:, :K] = m
        groups = ((m.view(-1, 4) != 0).sum(1) <= 2).all().item()
        assert ops.validate_24(m) == ops.validate_24(padded[:, :K]) == groups
