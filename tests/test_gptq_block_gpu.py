"""The column-block kernel where its variants meet: four to sixteen warps a block, safe and extreme divisors."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", [16, 32])
@pytest.mark.parametrize("rows", [4737, 9473, 20001])     # five and nine warps a block, more than one block of sixteen per SM
def test_rows_are_independent(cuda_device, rows, group):
    """One block of columns (no trailing update): parts of up to 4096 rows give the same bits as all rows together.  Some
    scales are so small or large that their warps take the IEEE divisions."""
    from fpq_b200 import ops

    g = torch.Generator(device=cuda_device).manual_seed(rows)
    x = torch.randn(512, 128, device=cuda_device, generator=g)
    H = x.t() @ x / 512
    U, status = ops.cholesky_inverse_upper(H)
    W = torch.randn(rows, 128, device=cuda_device, generator=g) * 0.02
    s = torch.rand(rows, 128 // group, device=cuda_device, generator=g) * 0.01 + 0.004
    s[5, 0], s[rows - 1, -1], s[4100] = 1e-33, 1e-35, 1e33
    whole = W.clone()
    codes = ops.gptq_quantize(whole, s, U, group)
    for lo in range(0, rows, 4096):
        part = W[lo:lo + 4096].clone()
        want = ops.gptq_quantize(part, s[lo:lo + 4096].contiguous(), U, group)
        assert torch.equal(codes[lo:lo + 4096], want) and torch.equal(whole[lo:lo + 4096], part)
    ops.check_device_errors(cuda_device)


def test_extreme_pivot_takes_the_general_division(cuda_device):
    """A factor whose diagonal leaves the range of the reciprocal form against the same factor a power of two smaller: the
    errors shrink exactly as the factor grows, so codes and weights agree."""
    from fpq_b200 import ops

    g = torch.Generator(device=cuda_device).manual_seed(0)
    U = torch.triu(torch.randn(128, 128, device=cuda_device, generator=g) * 0.05)
    U.diagonal().fill_(1.0)
    W = torch.randn(64, 128, device=cuda_device, generator=g)
    s = torch.rand(64, 8, device=cuda_device, generator=g) * 0.5 + 0.25
    a, b = W.clone(), W.clone()
    want = ops.gptq_quantize(a, s, U, 16)
    got = ops.gptq_quantize(b, s, U * 2.0 ** 101, 16)       # err / 2^101, times 2^101 U
    assert torch.equal(want, got) and torch.equal(a, b)


@pytest.mark.parametrize("cols", [1408, 2048])        # a ragged last group of blocks, whole groups
@pytest.mark.parametrize("group", [16, 32])
def test_slabs_of_rows_give_the_bits_of_the_whole(cuda_device, cols, group):
    """Many columns: the columns beyond a group are updated by one product where there are rows enough for the pair kernel, and
    block by block elsewhere (all 9473 rows: pairs for every group; 6344 of them: the first groups; 3000 and fewer:
    nowhere).  The codes and weights of a row must not depend on which."""
    from fpq_b200 import ops

    rows = 9473
    g = torch.Generator(device=cuda_device).manual_seed(cols)
    x = torch.randn(4 * cols, 32, device=cuda_device, generator=g) @ torch.randn(32, cols, device=cuda_device, generator=g) / 6
    x += torch.randn(4 * cols, cols, device=cuda_device, generator=g)
    H = x.t() @ x / (4 * cols)
    H.diagonal().add_(0.01)
    U, status = ops.cholesky_inverse_upper(H)
    assert int(status) == 0
    W = torch.randn(rows, cols, device=cuda_device, generator=g) * 0.02
    s = W.view(rows, cols // group, group).abs().amax(-1) / 6
    whole = W.clone()
    codes = ops.gptq_quantize(whole, s, U, group)
    for lo, hi in ((0, 3000), (3000, 3128), (3128, 3129), (3129, rows)):
        part = W[lo:hi].clone()
        want = ops.gptq_quantize(part, s[lo:hi].contiguous(), U, group)
        assert torch.equal(codes[lo:hi], want) and torch.equal(whole[lo:hi], part)
    ops.check_device_errors(cuda_device)
