"""The native host side of QuantizedLinear's forward: which calls it takes, and that the others go through the autograd
function as before."""
import pytest
import torch
import torch.autograd.forward_ad as fwad

from bitween_b200 import QuantizedLinear
from bitween_b200.kernels import _lib
from bitween_b200.modules import QuantizedLinearFunction

DEV = "cuda"


def test_calls_that_are_not_plain_are_left_to_the_python_path():
    forward = _lib.host_forward()
    x, q, s = torch.zeros(2, 64), torch.zeros(8, 8, dtype=torch.int32), torch.zeros(8, 2, dtype=torch.float16)
    assert forward(x, q, s, s, None, 4, 32) is None                    # not on a GPU
    assert forward(x, q, s, None, None, 4, 32) is None and forward(1, q, s, s, None, 4, 32) is None
    assert forward(x, q, s, s, None, 4.0, 32) is None and forward(x, q, s, s, None, 4, 1 << 80) is None
    assert forward(x.to("meta"), q, s, s, None, 4, 32) is None
    with pytest.raises(TypeError):
        forward(x, q, s, s, None, 4)


def _linear(bits=4, g=32, bias=True):
    torch.manual_seed(bits + g)
    return QuantizedLinear.from_float(torch.nn.Linear(1024, 48, bias=bias).to(DEV), bits, g)


def _function(ql, x):
    return QuantizedLinearFunction.apply(x, ql.qweight, ql.scale, ql.zero_point, ql.bias, ql.bits, ql.group_size)


def _native(ql, x):
    return _lib.host_forward()(x, ql.qweight, ql.scale, ql.zero_point, ql.bias, ql.bits, ql.group_size)


@pytest.mark.gpu
@pytest.mark.parametrize("bits,g,bias", [(4, 32, True), (8, 128, False), (2, 64, True)])
def test_native_forward_equals_the_autograd_function(bits, g, bias):
    ql = _linear(bits, g, bias)
    for shape in ((1024,), (1, 1024), (5, 1024), (12, 1024), (30, 1024), (2, 3, 1024), (48, 1024), (1, 1, 1, 1024)):
        for dt in (torch.float16, torch.bfloat16, torch.float32):
            x = torch.randn(shape, device=DEV).to(dt)
            if len(shape) == 1:
                assert _native(ql, x).shape == (48,)
            with torch.no_grad():
                want = _function(ql, x)
                y = _native(ql, x)
                assert y is not None and torch.equal(y, want)        # (the stream's scratch is there by now where one is needed)
                got = ql(x)
            assert got.shape == want.shape == (*shape[:-1], 48) and got.dtype == torch.float16 and torch.equal(got, want)
    # in a capture: scratch of the graph's own, which is the Python path's
    x = torch.randn(12, 1024, device=DEV).half()
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(graph):
        assert _native(ql, x) is None
        got = ql(x)
    graph.replay()
    assert torch.equal(got, _function(ql, x))
    # on a side stream and in inference mode
    x = torch.randn(3, 1024, device=DEV).half()
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st), torch.inference_mode():
        y = ql(x)
    st.synchronize()
    assert torch.equal(y, _function(ql, x)) and y.is_inference()


@pytest.mark.gpu
def test_what_is_recorded_transformed_or_refused_stays_with_the_autograd_function():
    ql = _linear()
    x = torch.randn(3, 1024, device=DEV).half()
    assert _native(ql, x) is not None
    # gradients
    xr = x.clone().requires_grad_(True)
    assert _native(ql, xr) is None
    y = ql(xr)
    assert y.grad_fn is not None and type(y.grad_fn).__name__ == "QuantizedLinearFunctionBackward"
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t, lambda t: t):
        ql(xr).sum().backward()
    assert len(packed) == 5 and xr.grad is not None
    with torch.no_grad():
        assert _native(ql, xr) is not None and not ql(xr).requires_grad
    ql.scale.requires_grad_(True)
    assert _native(ql, x) is None and ql(x).requires_grad
    ql.scale.requires_grad_(False)
    # forward-mode tangents, transforms, tracing, modes, subclasses
    with fwad.dual_level():
        dual = fwad.make_dual(x, torch.ones_like(x))
        with torch.no_grad():
            assert _native(ql, dual) is None
    seen = []
    for transform in (torch.func.vmap, lambda f: (lambda a: torch.func.grad(lambda b: (f(b), b.sum().float())[1])(a))):
        try:
            transform(lambda a: (seen.append(_native(ql, x)), a * 1)[1])(x)
        except Exception:      # noqa: BLE001 -- what matters is what the native call answered inside
            pass
    assert seen and all(r is None for r in seen)
    assert torch.jit.trace(lambda a: (seen.append(_native(ql, a)), a * 1)[1], x, check_trace=False) is not None and seen[-1] is None

    class Sub(torch.Tensor):
        pass

    assert _native(ql, x.as_subclass(Sub)) is None
    from torch.utils._python_dispatch import TorchDispatchMode

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    with Mode():
        assert _native(ql, x) is None
    # layouts and types that are converted, and what is refused
    assert _native(ql, torch.randn(1024, 3, device=DEV).half().t()) is None and _native(ql, x.double()) is None
    assert torch.equal(ql(x.double()), ql(x)) and torch.equal(ql(x.t().contiguous().t()), ql(x))
    for bad in (x[:, :128].contiguous(), torch.randn(3, 128, device=DEV)):
        assert _native(ql, bad) is None
        with pytest.raises(ValueError):
            ql(bad)
    with pytest.raises(RuntimeError):
        ql(x.cpu())
    empty = ql(x[:0])
    assert _native(ql, x[:0]) is None and empty.shape == (0, 48)
