"""The one-call forward and the direct training calls against the general path, over the forms of input both accept."""
import pytest
import torch

from fpq_b200.fp_quant import FPQuantConfig, FPQuantDtype, FPQuantLinear
from fpq_b200.fp_quant.module import linear_fns

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
                assert (fused(x) is not None) == (transform != "gsr" and bias is not torch.float32)
                layer._fused_forward = lambda *a: None
                want = layer(x)
                layer._fused_forward = fused
                assert got.shape == want.shape and got.dtype == want.dtype and torch.equal(got, want)
            if method == "abs_max" and transform != "gsr":
                for m in (1, 65, 300):
                    g, u = base[:m], torch.randn(m, k, device=cuda_device).bfloat16()
                    got = layer.forward_silu_mul(g, u)
                    assert (fused(g, u) is not None) == (bias is not torch.float32)
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
def test_training_matches_the_general_path(cuda_device, monkeypatch, fmt, backward, method, group, tokens):
    """Same kernels on the same operands: output and gradients bit for bit."""
    k, n = 384, 256
    layer = _layer(cuda_device, k, n, fmt, method, group, torch.bfloat16, backward=backward, master=True)
    x = torch.randn(*tokens, k, device=cuda_device).bfloat16()
    g = torch.randn(*tokens, n, device=cuda_device).bfloat16() * 0.01
    out, direct = [], []
    training_forward = linear_fns._training_forward

    def watch(*args, **kwargs):
        result = training_forward(*args, **kwargs)
        direct.append(result[3])
        return result

    monkeypatch.setattr(linear_fns, "_training_forward", watch)
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
    # the kernels directly, then the registered ops; the MXFP4 backward reads swizzled scales up to a rotation of 32 alone
    assert direct == ([] if backward == "BF16" else [not (backward == "MXFP4" and group > 32), False])


@pytest.mark.parametrize("backward", ["MXFP8", "MXFP4"])
@pytest.mark.parametrize("group", [32, 64])
def test_rotation_of_fp32_layers_is_classified_once_a_pass(cuda_device, monkeypatch, backward, group):
    """A matrix that has to be converted to bf16 is a new tensor on every pass, and classifying it waits for the GPU: at most one
    wait in the forward and one in the backward, whatever path the rotation takes."""
    from fpq_b200 import rotation

    layer = _layer(cuda_device, 384, 256, "MXFP4", "quest", group, backward=backward, master=True, dtype=torch.float32)
    x = torch.randn(64, 384, device=cuda_device, requires_grad=True)
    layer(x).sum().backward()
    waits = []
    sylvester = rotation.sylvester
    monkeypatch.setattr(rotation, "sylvester", lambda g: (waits.append(g), sylvester(g))[1])
    y = layer(x)
    assert len(waits) <= 1
    y.sum().backward()
    assert len(waits) <= 2


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


def test_graphs_outlive_other_streams(cuda_device):
    """A graph per stream, each after a warm-up on that stream, then passes on yet other streams: replays of every graph still
    read the tensor scales that they were captured with, although the memory of whatever was dropped has been reused."""
    layer = _layer(cuda_device, 384, 256, "NVFP4", "abs_max", 16, torch.bfloat16)
    x = torch.randn(40, 384, device=cuda_device).bfloat16()
    graphs, streams = [], []
    with torch.no_grad():
        want = layer(x).clone()
        for _ in range(10):
            stream = torch.cuda.Stream()
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                layer(x)
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                y = layer(x)
            graphs.append((graph, y))
            streams.append(stream)
            with torch.cuda.stream(stream):             # takes up whatever small blocks this stream's sets left
                streams.append([torch.full((1,), 1e4, device=cuda_device) for _ in range(40)])
        streams.append([torch.full((1,), 1e4, device=cuda_device) for _ in range(200)])
        for graph, y in graphs:
            y.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, want)


@pytest.mark.parametrize("fmt,backward", [("MXFP4", "MXFP8"), ("MXFP4", "MXFP4"), ("NVFP4", "BF16")])
def test_replayed_training_steps_follow_the_tensor_scales(cuda_device, fmt, backward):
    """A graph of a training step derives what it needs from the two tensor scales itself: a replay after an update in place
    gives what an eager step gives."""
    k, n = 384, 256
    layer = _layer(cuda_device, k, n, fmt, "abs_max", 16 if fmt == "NVFP4" else 32, None, backward=backward, master=True)
    x = torch.randn(128, k, device=cuda_device).bfloat16().requires_grad_(True)
    g = torch.randn(128, n, device=cuda_device).bfloat16() * 0.01

    def step():
        return torch.autograd.grad((y := layer(x)), (x, layer.weight), g) + (y.detach(),)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    with torch.no_grad():
        layer.weight_global_scale.mul_(0.5)
        layer.act_global_scale.mul_(0.25)
    want = step()
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(out, want):
        assert torch.equal(a, b)
