"""The one-call forward and the direct training calls against the general path, over the forms of input both accept."""
import pytest
import torch

from fpq_b200.fp_quant import FPQuantConfig, FPQuantDtype, FPQuantLinear

pytestmark = pytest.mark.gpu


def _layer(dev, k, n, fmt, method="abs_max", group=32, bias=None, transform="hadamard", backward="BF16", master=False, dtype=torch.bfloat16):
    torch.manual_seed(k + n)
    cfg = FPQuantConfig(forward_dtype=FPQuantDtype[fmt], forward_method=method, backward_dtype=FPQuantDtype[backward],
                        store_master_weights=master, hadamard_group_size=group, transform_init=transform)
    layer = FPQuantLinear(k, n, cfg, bias=bias is not None, device=dev, dtype=dtype)
    with torch.no_grad():
        layer.weight.normal_(0, 0.02)
        if bias is not None:
            layer.bias.normal_(0, 0.1)
    layer.pre_forward()
    if bias is not None:
        layer.bias = torch.nn.Parameter(layer.bias.detach().to(bias))
    return layer


@pytest.mark.parametrize("fmt,method,group,transform", [("MXFP4", "abs_max", 32, "hadamard"), ("MXFP4", "quest", 64, "hadamard"),
                                                        ("NVFP4", "abs_max", 16, "hadamard"), ("NVFP4", "abs_max", 128, "identity"),
                                                        ("MXFP4", "abs_max", 32, "gsr")])
@pytest.mark.parametrize("k,n", [(384, 256), (1024, 136)])     # 384: scale columns padded to a multiple of four for MXFP4 and exact for NVFP4
def test_inference_matches_the_general_path(cuda_device, fmt, method, group, transform, k, n):
    for bias in (None, torch.bfloat16, torch.float32):
        layer = _layer(cuda_device, k, n, fmt, method, group, bias, transform)
        base = torch.randn(300, k, device=cuda_device).bfloat16()
        forms = [base[:1], base[:64], base[:129], base, base[:6].view(2, 3, k), base[::2], base[:8].float(),
                 base[:8].half(), base.t().contiguous().t()[:40]]
        with torch.no_grad():
            for x in forms:
                got = layer(x)
                fused = layer._fused_forward
                layer._fused_forward = lambda *a: None
                want = layer(x)
                layer._fused_forward = fused
                assert got.shape == want.shape and got.dtype == want.dtype and torch.equal(got, want)
            if method == "abs_max" and transform != "gsr":
                for m in (1, 65, 300):
                    g, u = base[:m], torch.randn(m, k, device=cuda_device).bfloat16()
                    got = layer.forward_silu_mul(g, u)
                    layer._fused_forward = lambda *a: None
                    want = layer.forward_silu_mul(g, u)
                    layer._fused_forward = fused
                    assert torch.equal(got, want)
            with pytest.raises(Exception):
                layer(base[:, : k // 2])
            with pytest.raises(Exception):
                layer(base[0])
    # a changed tensor scale and a replaced weight are seen
    with torch.no_grad():
        layer = _layer(cuda_device, k, n, fmt, method, group, None, transform)
        y0 = layer(base)
        layer.weight_global_scale.mul_(2)
        y1 = layer(base)
        assert torch.allclose(y1.float() * 2, y0.float(), rtol=2e-2, atol=1e-3) and not torch.equal(y0, y1)


@pytest.mark.parametrize("fmt,backward,method,group", [("MXFP4", "MXFP8", "abs_max", 32), ("MXFP4", "MXFP8", "quest", 32),
                                                       ("MXFP4", "MXFP4", "quest", 32), ("MXFP4", "MXFP4", "abs_max", 64),
                                                       ("NVFP4", "BF16", "abs_max", 16), ("MXFP4", "BF16", "quest", 32)])
@pytest.mark.parametrize("tokens", [(64,), (2, 77)])
def test_training_matches_the_general_path(cuda_device, fmt, backward, method, group, tokens):
    """Same kernels on the same operands: output and gradients bit for bit."""
    k, n = 384, 256
    layer = _layer(cuda_device, k, n, fmt, method, group, torch.bfloat16, backward=backward, master=True)
    x = torch.randn(*tokens, k, device=cuda_device).bfloat16()
    g = torch.randn(*tokens, n, device=cuda_device).bfloat16() * 0.01
    out = []
    for general in (False, True):
        if general:
            layer._training_constants = lambda x: None
        xi = x.clone().requires_grad_(True)
        layer.weight.grad = layer.bias.grad = None
        y = layer(xi)
        y.backward(g)
        out.append((y, xi.grad, layer.weight.grad, layer.bias.grad))
    for a, b in zip(*out):
        assert torch.equal(a, b)


def test_long_products_and_other_streams(cuda_device):
    """Above the size where quantise and GEMM become two calls; passes on a stream of their own and from a graph that was
    captured before any eager pass."""
    k, n, m = 1024, 8192, 18000
    for fmt, method, group in (("MXFP4", "quest", 32), ("NVFP4", "abs_max", 16)):
        layer = _layer(cuda_device, k, n, fmt, method, group, torch.bfloat16)
        x = torch.randn(m, k, device=cuda_device).bfloat16()
        with torch.no_grad():
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            layer._blocked_weight_scales()
            from fpq_b200 import ops
            ops.device_error_flag(cuda_device)
            warm = _layer(cuda_device, k, n, fmt, method, group, torch.bfloat16)
            warm(x), warm(x[:100])
            torch.cuda.synchronize()
            with torch.cuda.graph(graph):
                captured = layer(x[:100])
            got, small = layer(x), layer(x[:100])
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(captured, small) and torch.equal(got[:100], small)
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                other = layer(x[:100])
            side.synchronize()
            assert torch.equal(other, small)
            fused = layer._fused_forward
            layer._fused_forward = lambda *a: None
            assert torch.equal(layer(x), got)
            layer._fused_forward = fused
