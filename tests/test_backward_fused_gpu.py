"""Fused kernels of the quantised backward passes against the CPU oracle."""
import pytest
import torch

from oracle import fp4

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", [0, 16, 32, 64, 128])
@pytest.mark.parametrize("rows", [1, 37, 2500])     # less than one warp's chunks, ragged, more than one per thread
def test_masked_rotation_matches_the_oracle(cuda_device, group, rows):
    """rotate(x .* mask): bit-exact, since both are the fp32 butterfly of the masked bf16 values, rounded once."""
    from fpq_b200 import ops

    cols = 384
    g = torch.Generator().manual_seed(rows + group)
    x = torch.randn(rows, cols, generator=g).bfloat16()
    mask = torch.rand(rows, cols, generator=g) < 0.9
    packed = fp4.pack_clip_mask(mask)
    y = x.float() * mask
    want = (fp4.fwht_butterfly(y, group) if group else y).bfloat16()
    got = ops.rotate_hadamard_masked(x.to(cuda_device), packed.to(cuda_device), group)
    assert torch.equal(got.cpu(), want)
    x[0, 5] = float("inf")                           # not hidden by a zero bit: inf * 0 = NaN
    mask[0, 5] = False
    got = ops.rotate_hadamard_masked(x.to(cuda_device), fp4.pack_clip_mask(mask).to(cuda_device), group)
    assert bool(got[0, 5].isnan())


@pytest.mark.parametrize("group", [0, 16, 32])
@pytest.mark.parametrize("rows,cols", [(1, 32), (37, 96), (128, 64), (161, 1056), (2500, 384)])   # part of a tile, ragged runs
def test_requantized_transpose_matches_the_two_steps(cuda_device, group, rows, cols):
    """MXFP4 -> dequantise, transpose, rotate, quantise in one pass: the same bytes as the two kernels it stands for (the
    transposing dequantiser and the quantiser, each pinned to the oracle), for ordinary and extreme scales and divisors,
    either scale layout on both sides."""
    from fpq_b200 import ops

    g = torch.Generator().manual_seed(rows * 3 + group)
    codes = torch.randint(0, 256, (rows, cols // 2), generator=g, dtype=torch.uint8).to(cuda_device)
    sb = torch.randint(120, 134, (rows, cols // 32), generator=g, dtype=torch.uint8)
    for alpha, extreme in ((3.0, False), (1.0, True), (2e6, False), (1e-7, False), (0.37, True)):
        s = sb.clone()
        if extreme:
            s[torch.rand(s.shape, generator=g) < 0.2] = 20          # beyond the table's exponent range
            s[torch.rand(s.shape, generator=g) < 0.1] = 235
            s[0, 0] = 0
        s = s.to(cuda_device)
        al = torch.tensor([alpha], device=cuda_device)
        xt = ops.mxfp4_transpose_dequant(codes, s, al, pad_to=32)
        want_q, want_s, _ = ops.quantize(xt, "mxfp4", group)
        got_q, got_s = ops.mxfp4_requantize_transposed(codes, s, al, group)
        assert torch.equal(got_q, want_q) and torch.equal(got_s, want_s)
        q2, s2 = ops.mxfp4_requantize_transposed(codes, ops.swizzle_scales(s), al, group, swizzled=True, scales_swizzled=True)
        assert torch.equal(q2, want_q) and torch.equal(s2, ops.swizzle_scales(want_s))


@pytest.mark.parametrize("t,n", [(1, 8), (33, 40), (96, 264), (1000, 1032)])
def test_transposed_quantiser_at_ragged_runs(cuda_device, t, n):
    """The bf16 form where the last run of tiles along t is short and the last column tile ragged: the bytes of the quantiser
    on the padded transposed copy."""
    from fpq_b200 import ops

    x = torch.randn(t, n, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(t)).bfloat16()
    tp = -(-t // 128) * 128
    xt = torch.zeros(n, tp, dtype=torch.bfloat16, device=cuda_device)
    xt[:, :t] = x.t()
    want_q, want_s, _ = ops.quantize(xt, "mxfp4", 32)
    got_q, got_s = ops.quantize_transposed(x, 32, pad_to=128)
    assert torch.equal(got_q, want_q) and torch.equal(got_s, want_s)
