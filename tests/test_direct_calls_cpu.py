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


def _yes():
    return True


def _no():
    return False


def test_a_captured_graphs_constants_outlive_other_streams_and_new_scales():
    """What a captured inference pass was given stays alive with the cache and at its address, whatever streams and scales
    come after, and holds the values of new scales once a pass has seen them on the set's stream."""
    w, a = _scales()
    cache = ConstantsCache()
    own = cache.inference(w, a, 1, _no)
    assert cache.inference(w, a, 1, _yes) is own and cache.inference(w, a, 2, _yes) is own     # its own stream's, another's
    held, address = weakref.ref(own), [t.data_ptr() for t in (own.alpha, own.act_scale, own.weight_scale)]
    del own
    for stream in range(2, cache.STREAMS + 16):
        assert float(cache.inference(w, a, stream, _no).alpha) == float((1.0 / (w * a)).float())
    assert len(cache._inference) == cache.STREAMS
    w.mul_(2)
    fresh = cache.inference(w, a, 1, _yes)                 # no set of the new scales yet: the graph's own
    assert fresh is not held() and float(held().weight_scale) == 3.0
    other = torch.tensor([5.0], dtype=torch.bfloat16)
    for scale in (w, other):
        for stream in range(1, cache.STREAMS + 16):
            got = cache.inference(scale, a, stream, _no)
            assert float(got.weight_scale) == float(scale) and float(got.alpha) == float((1.0 / (scale * a)).float())
        assert cache.inference(scale, a, 1, _no) is held() and float(held().weight_scale) == float(scale)
    assert [t.data_ptr() for t in (held().alpha, held().act_scale, held().weight_scale)] == address


def test_sets_do_not_write_into_fp32_scales():
    w, a = torch.tensor([3.0]), torch.tensor([2.0])
    cache = ConstantsCache()
    cache.inference(w, a, 1, _no)
    other = torch.tensor([7.0])
    assert float(cache.inference(other, a, 1, _no).weight_scale) == 7.0
    assert float(w) == 3.0


def test_what_a_capture_makes_is_not_kept():
    w, a = _scales()
    cache = ConstantsCache()
    first = cache.inference(w, a, 1, _yes)                 # no earlier pass: made inside the graph
    assert cache.inference(w, a, 1, _no) is not first
    eager = cache.training(w, a, 1, False)
    follow = cache.training(w, a, 1, True)                 # a training step's graph derives its own
    assert follow is not eager and cache.training(w, a, 1, False) is eager


def test_training_constants_follow_the_scales_and_stay_as_they_are():
    w, a = _scales()
    cache = ConstantsCache()
    first = cache.training(w, a, 1, False)
    assert cache.training(w, a, 1, False) is first
    a.mul_(0.5)
    second = cache.training(w, a, 1, False)
    assert second is not first and float(second.act_scale) == 1.5 and float(first.act_scale) == 3.0
    other = w.clone()
    assert cache.training(other, a, 1, False) is not second     # another object, equal values
    errors = []

    def passes(scale):
        try:
            mine = torch.tensor([scale], dtype=torch.bfloat16)
            for i in range(300):
                got = cache.training(mine if i % 3 else other, a, i % (cache.STREAMS + 3), False)
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
    twin = copy.deepcopy(layer)
    assert not twin._constants._inference and float(twin._gemm_alpha()) == want
    del layer._constants
    loaded = pickle.loads(pickle.dumps(layer))
    assert float(loaded._gemm_alpha()) == want
