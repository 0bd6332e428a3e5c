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
