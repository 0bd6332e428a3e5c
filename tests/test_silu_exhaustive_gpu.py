"""The fused SiLU against torch's on every bf16 gate: those of the fast form (up to 80) one by one, beyond them by chunks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_silu_matches_torch_on_every_gate(cuda_device):
    """Row per gate g: element 0 is silu(g) * 2^k, element 16 is minus torch's silu(g) * 2^k (made with the gate 64, whose
    silu is 64).  After the Hadamard rotation of 32 the first NVFP4 group holds only their difference, so its scale byte is
    zero exactly when the two bf16 values are the same; a difference of one bf16 unit gives a non-zero byte."""
    from fpq_b200 import ops

    bits = torch.arange(65536, dtype=torch.int32).to(torch.int16)
    g = bits.view(torch.bfloat16).to(cuda_device)
    want = torch.nn.functional.silu(g)
    g = g[g.abs() <= 80]                # all gates of the fast form, zeros and subnormal ones among them
    want = torch.nn.functional.silu(g)
    k = -torch.floor(torch.log2(want.float().abs())).clamp(-120, 120)
    up = torch.exp2(k).bfloat16()
    gs = torch.tensor([2.0 ** 14], device=cuda_device)

    def scale_bytes(reference):
        gate, upm = torch.zeros(2, g.numel(), 32, dtype=torch.bfloat16, device=cuda_device)
        gate[:, 0], upm[:, 0] = g, up
        gate[:, 16], upm[:, 16] = 64.0, -(reference.float() * up.float() / 64).bfloat16()
        return ops.quantize_silu_mul(gate, upm, "nvfp4", 32, gs, swizzled=False)[1]

    sb = scale_bytes(want)
    assert g.numel() == 2 * (0x42a0 + 1) and not bool(sb[:, 0].any())
    assert bool((sb[:, 1] != 0)[want != 0].all())
    off = (want.view(torch.int16) + 1).view(torch.bfloat16)
    assert bool((scale_bytes(off)[:, 0] != 0).all())


def test_gates_out_of_the_fast_range(cuda_device):
    """Chunks with a gate beyond +-80, an infinity or a NaN take the library exponential: the two-step result."""
    from fpq_b200 import ops

    gate = torch.randn(64, 256, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(1)).bfloat16()
    up = torch.randn_like(gate)
    for i, v in enumerate([80.0, -80.0, 80.5, -80.5, -88.5, -100.0, 3e38, -3e38, float("inf"), float("nan"), 1e-40, -0.0]):
        gate[i, 7 * i % 256] = v
    q, sb = ops.quantize_silu_mul(gate, up, "mxfp4", 32, None, swizzled=False)
    q2, sb2, _ = ops.quantize(torch.nn.functional.silu(gate) * up, "mxfp4", 32, None)
    assert torch.equal(q, q2) and torch.equal(sb, sb2)
