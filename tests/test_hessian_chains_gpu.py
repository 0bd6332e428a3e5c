"""The accumulation chains and tile bands of the Hessian / A^T B kernel where they can go wrong: a chain of one token,
ragged last chains, one to many bands, tiles beyond the matrix, an output whose rows are not 32-byte aligned."""
import numpy as np
import pytest
import torch

from tests import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,d", [
    (4097, 3080),        # pair kernel, second chain of one token, ragged edge tiles, two bands
    (8192 + 4032, 4104), # three chains, 17 block rows: the last band is one row high, one column block of 8
    (20000, 3072),       # five chains, one more than a whole number of bands
    (9000, 1032),        # single-CTA kernel: one launch per chain
])
def test_chains_match_fp64(cuda_device, tokens, d):
    """1e-5 relative Frobenius as for a single chain: chains are added with rounded fp32 additions (2^-24 each)."""
    from fpq_b200 import ops

    x = inputs.correlated_activations(tokens, d, seed=tokens).to(cuda_device)
    h0 = torch.randn(d, d, device=cuda_device)
    h0 = h0 + h0.t()
    H = h0.clone()
    ops.hessian_accumulate(H, x, alpha=0.5, beta=0.25)
    ops.check_device_errors(cuda_device)
    want = 0.25 * h0.double() + 0.5 * (x.double().t() @ x.double())
    assert ((H.double() - want).norm() / want.norm()).item() < 1e-5
    assert torch.equal(H, H.t())


@pytest.mark.parametrize("tokens,d", [(4097, 3080), (8192 + 4032, 4104), (12288, 3072)])
@pytest.mark.parametrize("beta", [0.0, 0.25])
def test_one_update_is_chain_by_chain(cuda_device, tokens, d, beta):
    """The bits of one update are those of its chains of 4096 tokens applied one after the other, each addition rounded into
    the output: how far a run is split must not show in the Hessian."""
    from fpq_b200 import ops

    x = inputs.correlated_activations(tokens, d, seed=d).to(cuda_device)
    h0 = torch.randn(d, d, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(d))
    h0 = h0 + h0.t()
    got, want = h0.clone(), h0.clone()
    ops.hessian_accumulate(got, x, alpha=0.3, beta=beta)
    for t in range(0, tokens, 4096):
        ops.hessian_accumulate(want, x[t:t + 4096], alpha=0.3, beta=beta if t == 0 else 1.0)
    ops.check_device_errors(cuda_device)
    assert torch.equal(got, want)


def test_output_rows_off_the_vector_alignment(cuda_device):
    """d = 3724: rows of 14896 bytes, not a multiple of 32; the trailing updates run on CTA pairs (big enough) and take
    the element-wise store.  fp32 chain: residual of U^T U H below 1e-3 for a Hessian of condition < 1e3."""
    from fpq_b200 import ops

    d = 3724
    x = torch.randn(2 * d, d, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(3))
    H = x.t() @ x / d
    H.diagonal().add_(0.1)
    U, status = ops.cholesky_inverse_upper(H)
    ops.check_device_errors(cuda_device)
    assert int(status) == 0
    r = U.double().t() @ (U.double() @ H.double()) - torch.eye(d, device=cuda_device, dtype=torch.float64)
    assert r.abs().max().item() < 1e-3


@pytest.mark.parametrize("d", [1, 31, 33, 127, 128, 129, 160, 257, 300, 640, 1100])
def test_factor_at_block_edges(cuda_device, d):
    """U = chol(H^-1, upper) where the 128-blocks, the 32-column blocks inside them and the 32-row panels end raggedly.  The
    chain is backward stable: with a condition number of a few hundred and d eps = 7e-5 at most, 1e-4 relative holds with room."""
    from fpq_b200 import ops

    x = torch.randn(2 * d + 8, d, device=cuda_device, dtype=torch.float64, generator=torch.Generator(device=cuda_device).manual_seed(d))
    H = x.t() @ x / (2 * d)
    H.diagonal().add_(0.05)
    U, status = ops.cholesky_inverse_upper(H.float())
    want = torch.linalg.cholesky(torch.linalg.inv(H.float().double()), upper=True)
    ops.check_device_errors(cuda_device)
    assert int(status) == 0 and not bool(torch.tril(U, -1).any())
    assert ((U.double() - want).norm() / want.norm()).item() < 1e-4


def test_bad_pivots_are_reported(cuda_device):
    from fpq_b200 import ops

    for i, v in ((0, 0.0), (40, -1.0), (127, float("nan")), (130, float("inf"))):
        H = torch.eye(200, device=cuda_device)
        H[i, i] = v
        U, status = ops.cholesky_inverse_upper(H)
        assert int(status) == 1
    ops.check_device_errors(cuda_device)


def _fma(a, b, c):
    """fl32(a * b + c) of float32 arrays, rounded once: the product is exact in fp64, the sum is rounded to odd there."""
    prod = a.astype(np.float64) * b.astype(np.float64)
    c = c.astype(np.float64)
    s = prod + c
    t = s - prod
    err = (prod - (s - t)) + (c - t)
    bits = s.view(np.int64)
    step = np.where((err > 0) == (s > 0), 1, -1)
    return np.where((err != 0) & (bits & 1 == 0), bits + step, bits).view(np.float64).astype(np.float32)


@pytest.mark.parametrize("d", [128, 100, 33, 1])
def test_diagonal_block_is_right_looking_elimination(cuda_device, d):
    """One block: bit for bit the elimination column by column, A[i, j] = fma(-c_i, c_j / pivot, .) and the same for the rows of
    the inverse, whatever order the kernel works in (1 / sqrt(pivot) from the device's rsqrt and one Newton step)."""
    from fpq_b200 import ops

    x = torch.randn(2 * d + 8, d, generator=torch.Generator().manual_seed(d))
    H = x.t() @ x / (2 * d)
    H.diagonal().add_(0.05)
    U, status = ops.cholesky_inverse_upper(H.to(cuda_device))
    assert int(status) == 0
    a = H.numpy()[::-1, ::-1].copy()
    inv = np.eye(d, dtype=np.float32)
    out = np.zeros((d, d), dtype=np.float32)
    for k in range(d):
        c, piv = a[:, k].copy(), a[k, k]
        rec = np.float32(1) / piv
        low = slice(k + 1, d)
        a[low, low] = _fma(-c[low, None] + 0 * a[low, low], (c[low] * rec)[None, :] + 0 * a[low, low], a[low, low])
        inv[low] = _fma(-c[low, None] + 0 * inv[low], (inv[k] * rec)[None, :] + 0 * inv[low], inv[low])
        r = torch.rsqrt(torch.tensor([piv], device=cuda_device)).cpu().numpy()
        r = r * _fma((np.float32(-0.5) * piv) * r, r, np.full(1, 1.5, np.float32))
        out[k] = inv[k] * r[0]
    assert np.array_equal(U.cpu().numpy()[::-1, ::-1], out)


def test_largest_and_smallest_pivots(cuda_device):
    """Pivots near the ends of fp32, whose reciprocals are subnormal or nearly overflow, are eliminated like any other."""
    from fpq_b200 import ops

    d = 200
    for big, c in ((2e38, 2e19), (9e37, 1e19), (8e-39, 4e-20)):
        for i in (150, 60):                          # in the first and the second block
            H = 10 * torch.eye(d, dtype=torch.float64)
            H[i, i] = big
            H[i, 3] = H[3, i] = c                    # rows are eliminated from the last to the first
            H = H.float()
            low = torch.linalg.cholesky(H.double().flip(0, 1))
            want = torch.linalg.solve_triangular(low, torch.eye(d, dtype=torch.float64), upper=False).flip(0, 1)
            U, status = ops.cholesky_inverse_upper(H.to(cuda_device))
            assert int(status) == 0
            # 1 / 2e38 as a subnormal has 21 bits
            assert torch.allclose(U.cpu().double(), want, rtol=2e-6, atol=0)
