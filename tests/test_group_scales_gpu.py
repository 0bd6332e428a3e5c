"""The element-wise steps of round-to-nearest at the values where they can go wrong."""
import pytest
import torch

from oracle import fp4

pytestmark = pytest.mark.gpu

EXTREME = [0.0, -0.0, 1e-45, -1e-39, 1e-30, 0.25, -0.75, 1.25, 1.75, 2.5, 3.5, 5.0, 6.0, 1e20, -3e38, float("inf"), -float("inf"), float("nan")]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("group", [16, 32, 24, 4])
def test_apply_scales_at_the_edges(cuda_device, dtype, group):
    """Grid values, codes and dequantised values = the grid value nearest to the IEEE quotient: on the CPU in the same
    fp32 operations.  Shared and separate scales, every pairing of extreme values and scales, quotients next to every
    rounding boundary."""
    from fpq_b200 import _cabi as C
    from fpq_b200 import ops

    rows, cols = 64, 96
    g = torch.Generator().manual_seed(group)
    x = torch.randn(rows, cols, generator=g) * 4
    s = torch.rand(rows, cols // group, generator=g) + 0.01
    edge = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0]).repeat_interleave(3)
    ulps = torch.tensor([-1, 0, 1]).repeat(7).int()
    edge = (edge.view(torch.int32) + ulps).view(torch.float32)
    for r in range(1, 20):
        x[r, : len(edge)] = edge * s[r].repeat_interleave(group)[: len(edge)]
    for r in range(20, 64):
        x[r, : len(EXTREME)] = torch.tensor(EXTREME)
        s[r] = [1.0, 1e-30, 1e30, 1e-38, 3e38, 1e-45, float("inf"), float("nan"), 0.0, -1.5, 0.37][r % 11]
    x = x.to(dtype)
    q = x.float() / s.repeat_interleave(group, dim=1)
    idx = sum((q.abs() > b if strict else q.abs() >= b).int() for b, strict in
              ((0.25, 1), (0.75, 0), (1.25, 1), (1.75, 0), (2.5, 1), (3.5, 0), (5.0, 1)))
    mag = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6.0])[idx]
    grid = torch.where((q < 0) | (idx == 0), -mag, mag)
    xd, sd = x.to(cuda_device), s.to(cuda_device)
    got = ops.apply_scales(xd, sd, group, C.OUT_GRID)
    assert torch.equal(got.cpu(), grid.to(dtype)) and torch.equal(got.cpu().signbit(), grid.signbit())
    want_codes = idx | ((grid.signbit()).int() << 3)
    want_codes = (want_codes[:, 0::2] | (want_codes[:, 1::2] << 4)).to(torch.uint8)
    assert torch.equal(ops.apply_scales(xd, sd, group, C.OUT_CODES).cpu(), want_codes)
    assert torch.equal(ops.pack_grid(got).cpu(), want_codes)
    dq = grid * s.repeat_interleave(group, dim=1)
    assert torch.equal(ops.apply_scales(xd, sd, group, C.OUT_DEQUANT).cpu().nan_to_num(7.0), dq.to(dtype).nan_to_num(7.0))
    if group % 8 == 0:
        m = ops.multiply_scales(got, sd.to(dtype), group)
        assert torch.equal(m.nan_to_num(7.0), (got * sd.to(dtype).repeat_interleave(group, dim=1)).nan_to_num(7.0))


@pytest.mark.parametrize("fmt", ["nvfp4", "mxfp4"])
def test_checks_of_the_scales(cuda_device, fmt):
    from fpq_b200.quantization.quantizer import Quantizer

    def make():
        nv = fmt == "nvfp4"
        return Quantizer(bits=4, symmetric=True, format="nvfp" if nv else "mxfp", granularity="group", group_size=16 if nv else 32,
                         scale_precision="e4m3" if nv else "e8m0")

    x = torch.randn(8, 64, device=cuda_device)
    scales, zeros = make().get_quantization_params(x)
    assert bool(scales.isfinite().all()) and not bool(zeros.any()) and zeros.shape == scales.shape
    q = make()
    grid = q.quantize(x, scales)
    assert torch.equal(q.dequantize(grid, scales), grid * scales.repeat_interleave(q.group_size, dim=1))
    if fmt == "nvfp4":
        with pytest.raises(ValueError, match="Global scale"):
            make().get_quantization_params(torch.zeros_like(x))
        q = make()
        q.deferred_checks = []
        q.get_quantization_params(torch.zeros_like(x))
        with pytest.raises(ValueError):
            q.raise_deferred_checks()
        # a NaN among the group scales, at once and deferred: no longer tracked, the tensor scale is not looked at itself
        for deferred in (False, True):
            q = make()
            q.get_quantization_params(x)
            q._track_global_scale = False
            q.global_scale.fill_(float("nan"))
            q.deferred_checks = [] if deferred else None
            with pytest.raises(ValueError, match="Scales"):
                q.get_quantization_params(x)
                q.raise_deferred_checks()


def test_dequantize_under_modes_and_transforms(cuda_device):
    """The product of `dequantize` where its kernel must not be called on an address: vmap, a dispatch mode that records it,
    make_fx, torch.compile without graph breaks and forward-mode derivatives."""
    import torch.autograd.forward_ad as forward_ad
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils._python_dispatch import TorchDispatchMode

    from fpq_b200.quantization.quantizer import Quantizer

    quantizer = Quantizer(bits=4, symmetric=True, format="mxfp", granularity="group", group_size=32, scale_precision="e8m0")
    q = torch.randint(-6, 7, (6, 96), device=cuda_device).float()
    s = torch.rand(6, 3, device=cuda_device) + 0.1
    want = q * s.repeat_interleave(32, dim=1)
    assert torch.equal(quantizer.dequantize(q, s), want)
    assert torch.equal(torch.func.vmap(quantizer.dequantize)(q.view(2, 3, 96), s.view(2, 3, 3)).view(6, 96), want)
    seen = []

    class Record(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    with Record():
        assert torch.equal(quantizer.dequantize(q, s), want)
    assert any("mul" in f for f in seen)
    traced = make_fx(lambda a, b: quantizer.dequantize(a, b))(q, s)
    assert torch.equal(traced(2 * q, s), 2 * want)
    assert torch.equal(torch.compile(quantizer.dequantize, backend="eager", fullgraph=True)(q, s), want)
    with forward_ad.dual_level():
        dual = quantizer.dequantize(forward_ad.make_dual(q, torch.ones_like(q)), s)
        tangent = forward_ad.unpack_dual(dual).tangent
        assert torch.equal(tangent, s.repeat_interleave(32, dim=1))
