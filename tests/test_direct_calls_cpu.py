"""When the native calls may be made on a tensor's address, and what a layer keeps between passes."""
import copy
import os
import pickle
import subprocess
import sys
import threading
import weakref

import torch
import torch.autograd.forward_ad as forward_ad
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

from fpq_b200.fp_quant.module.linear_fns import ConstantsCache
from fpq_b200.ops import plain_eager


class _Functions(TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


class _Dispatch(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


class _Subclass(torch.Tensor):
    pass


def test_plain_eager():
    x = torch.ones(2, 32)
    assert plain_eager(x) and plain_eager(torch.nn.Parameter(x))
    with torch.device("cpu"):                     # sets a default for factories, sees nothing else
        assert plain_eager(x)
    for mode in (_Functions(), _Dispatch(), forward_ad.dual_level()):
        with mode:
            assert not plain_eager(x)
    with torch.device("cpu"), _Functions():
        assert not plain_eager(x)
    assert not plain_eager(x.as_subclass(_Subclass))
    seen = []

    def look(t):
        seen.append(plain_eager(t))
        return t

    torch.func.vmap(look)(x)
    torch.func.jvp(look, (x,), (x,))
    torch.compile(look, backend="eager", fullgraph=True)(x)
    assert not any(seen) and len(seen) == 3


def test_another_torch_without_the_private_names():
    """The package loads, takes the general way and asks for the stream through the public call."""
    code = """
import sys, torch, types
for name in ("_len_torch_function_stack", "_cuda_getCurrentRawStream"):
    if hasattr(torch._C, name):
        delattr(torch._C, name)
from fpq_b200 import ops
assert not ops.plain_eager(torch.ones(2))
torch.cuda.current_stream = lambda device: types.SimpleNamespace(cuda_stream=(device, 7))
t = types.SimpleNamespace(device=torch.device("cuda", 1))
assert ops._stream(t) == (t.device, 7)
"""
    subprocess.run([sys.executable, "-c", code], check=True, env={**os.environ, "PYTHONPATH": os.pathsep.join(sys.path)})


def _scales():
    return torch.tensor([3.0], dtype=torch.bfloat16), torch.tensor([3.0], dtype=torch.bfloat16)


def test_a_captured_graphs_constants_outlive_other_streams_and_new_scales():
    """What a capture was given stays alive with the cache, whatever streams and scales come after."""
    w, a = _scales()
    cache = ConstantsCache()
    own = cache.get(w, a, 1, False)
    held = [weakref.ref(cache.get(w, a, 1, True)), weakref.ref(cache.get(w, a, 2, True))]     # its own stream's set, another's
    assert held[0]() is own and held[1]() is own
    kept = weakref.ref(cache.get(w, a, 3, False))
    del own
    for stream in range(4, 24):
        assert cache.get(w, a, stream, False) is cache.get(w, a, stream, False)
    w.mul_(2)
    for stream in range(1, 24):
        assert float(cache.get(w, a, stream, False).alpha) == float((1.0 / (w * a)).float())
    assert all(r() is not None for r in held) and kept() is None
    assert len(cache._of[3]) <= 8


def test_what_a_capture_makes_is_not_kept():
    w, a = _scales()
    cache = ConstantsCache()
    first = cache.get(w, a, 1, True)                       # no earlier pass: made inside the graph
    assert cache.get(w, a, 1, False) is not first
    eager = cache.get(w, a, 1, False)
    follow = cache.get(w, a, 1, True, follow=True)         # a training step's graph derives its own
    assert follow is not eager and cache.get(w, a, 1, False) is eager


def test_constants_follow_the_scales():
    w, a = _scales()
    cache = ConstantsCache()
    first = cache.get(w, a, 1, False)
    assert cache.get(w, a, 1, False) is first
    a.mul_(0.5)
    second = cache.get(w, a, 1, False)
    assert second is not first and float(second.act_scale) == 1.5
    other = w.clone()
    assert cache.get(other, a, 1, False) is not second     # another object, equal values
    errors = []

    def passes(scale):
        try:
            mine = torch.tensor([scale], dtype=torch.bfloat16)
            for i in range(300):
                got = cache.get(mine if i % 3 else other, a, i % 11, False)
                if float(got.weight_scale) != (scale if i % 3 else 3.0):
                    errors.append(i)
        except Exception as e:                              # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=passes, args=(float(2 ** i),)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


def test_layers_saved_without_constants_load():
    """A layer pickled whole before it kept constants, and a copy of a layer that has handed some to a capture."""
    from fpq_b200.fp_quant import FPQuantConfig, FPQuantDtype, FPQuantLinear

    layer = FPQuantLinear(64, 32, FPQuantConfig(forward_dtype=FPQuantDtype.MXFP4), device="cpu", dtype=torch.bfloat16)
    with torch.no_grad():
        layer.weight_global_scale.fill_(3)
        layer.act_global_scale.fill_(3)
    want = float(layer._gemm_alpha())
    layer._constants.get(layer.weight_global_scale, layer.act_global_scale, 0, True)
    twin = copy.deepcopy(layer)
    assert float(twin._gemm_alpha()) == want and not twin._constants._captured
    del layer._constants
    loaded = pickle.loads(pickle.dumps(layer))
    assert float(loaded._gemm_alpha()) == want
