"""The module's plain call (gn_python.cpp: plain_call, without views or inner ops) against the general path through the
ops, which a dispatch mode forces: values, sizes, strides, gradients, and what may surround a call."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

import channels_last_groupnorm_b200 as pkg

pytestmark = pytest.mark.gpu


class Pass(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def _order(t, order):
    """A tensor of t's sizes and values in the given storage order."""
    nd = t.ndim
    if order == "last":
        return t.permute(0, *range(2, nd), 1).contiguous().permute(0, nd - 1, *range(1, nd - 1))
    if order == "transposed":  # dense, but the spatial axes are swapped in memory
        return t.transpose(-1, -2).contiguous().transpose(-1, -2)
    if order == "gaps":
        return torch.cat([t, t], -1)[..., :t.shape[-1]]
    if order == "offset":  # storage that starts in the middle of 16 bytes
        flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)[1:]
        return flat.view(t.shape).copy_(t)
    return t.contiguous()


SHAPES = [(2, 32, 5, 7), (1, 24, 9, 3), (3, 16, 11), (2, 8, 3, 4, 5), (2, 8, 1, 1), (4, 8, 1), (1, 8, 1, 6), (3, 8, 6, 1), (2, 1, 4, 4), (1, 1, 1, 1)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("order", ["last", "first", "transposed", "gaps", "offset"])
@pytest.mark.parametrize("dtype,pdtype", [(torch.float16, torch.float16), (torch.bfloat16, torch.float32), (torch.float32, torch.float32),
                                          (torch.float64, torch.float64)], ids=lambda d: str(d)[6:])
def test_plain_call_equals_the_general_path(shape, order, dtype, pdtype):
    torch.manual_seed(3)
    groups = 4 if shape[1] > 1 else 1
    m = pkg.GN_NHWC(groups, shape[1], activation="silu", device="cuda", dtype=pdtype)
    with torch.no_grad():
        m.weight.normal_()
        m.bias.normal_()
    x = _order(torch.randn(shape, device="cuda").to(dtype), order).requires_grad_(True)
    inputs = (x, m.weight, m.bias)
    for dy_order in ("last", "first", "gaps"):
        dy = _order(torch.randn(shape, device="cuda").to(dtype), dy_order)
        got = m(x)
        grads = torch.autograd.grad(got, inputs, dy)
        with Pass():
            want = m(x)
            wgrads = torch.autograd.grad(want, inputs, dy)
        assert got.stride() == want.stride() and got.dtype == want.dtype and torch.equal(got, want)
        for a, b in zip(grads, wgrads):
            assert a.stride() == b.stride() and a.dtype == b.dtype and torch.equal(a, b)
    with torch.no_grad():
        y = m(x)
        assert torch.equal(y, want) and y.stride() == want.stride() and not y.requires_grad
    with torch.inference_mode():
        assert torch.equal(m(x), want) and m(x).is_inference()
    frozen = pkg.GN_NHWC(groups, shape[1], activation="silu", device="cuda", dtype=pdtype).requires_grad_(False)
    assert not frozen(x.detach()).requires_grad and frozen(x).requires_grad


def test_saved_tensors_on_the_cpu_double_backward_and_profiler():
    torch.manual_seed(4)
    m = pkg.GN_NHWC(4, 32, activation="gelu", device="cuda")
    x = _order(torch.randn(2, 32, 6, 5, device="cuda"), "last").requires_grad_(True)
    want = torch.autograd.grad(m(x).square().sum(), (x, m.weight, m.bias))
    with torch.autograd.graph.save_on_cpu():  # comes back in another storage order
        y = m(x)
    got = torch.autograd.grad(y.square().sum(), (x, m.weight, m.bias))
    assert all(torch.allclose(a, b, rtol=1e-5, atol=1e-5) for a, b in zip(got, want))  # (dy and x in channels-last order either way)
    with Pass():
        general = torch.autograd.grad(m(x).square().sum(), (x, m.weight, m.bias), create_graph=True)
    plain = torch.autograd.grad(m(x).square().sum(), (x, m.weight, m.bias), create_graph=True)
    for a, b in zip(plain, general):
        assert torch.equal(a, b) and a.requires_grad == b.requires_grad
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        m(x).sum().backward()
    names = {e.key for e in prof.key_averages()}
    assert any("gnb200::fwd" in n for n in names) and any("gnb200::bwd" in n for n in names)


def test_what_is_refused_stays_refused():
    m = pkg.GN_NHWC(4, 32, device="cuda")
    for bad in (torch.randn(2, 16, 4, 4, device="cuda"), torch.randn(2, 32, device="cuda"), torch.randn(2, 32, 4, 4)):
        with pytest.raises(ValueError):
            m(bad)
    x = torch.randn(2, 32, 4, 4, device="cuda")
    for bad in (torch.randint(0, 9, (2, 32, 4, 4), device="cuda"), x.bool()):
        with pytest.raises(RuntimeError):
            m(bad)
    m.num_groups = 5
    with pytest.raises(RuntimeError, match="divisible"):
        m(x)
    with pytest.raises(RuntimeError):  # an empty batch
        pkg.GN_NHWC(4, 32, device="cuda")(x[:0])
    assert pkg.GN_NHWC(4, 32, affine=False)(x).shape == x.shape


def test_function_modes_and_subclasses_see_the_call():
    m = pkg.GN_NHWC(4, 32, device="cuda")
    x = torch.randn(2, 32, 4, 4, device="cuda")
    seen = []

    class Log(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    with Log():
        y = m(x)
    assert any("group_norm_act" in s for s in seen) and torch.equal(y, m(x))

    class Sub(torch.Tensor):
        pass

    assert type(m(x.as_subclass(Sub))) is Sub or torch.equal(m(x.as_subclass(Sub)), y)


def test_subclasses_are_no_plain_calls():
    class Sub(torch.Tensor):
        seen = []

        @classmethod
        def __torch_function__(cls, func, types, args=(), kwargs=None):
            cls.seen.append(func)
            return super().__torch_function__(func, types, args, kwargs or {})

    m = pkg.GN_NHWC(4, 32, device="cuda")
    x = torch.randn(2, 32, 4, 4, device="cuda")
    y = m(x)
    assert not Sub.seen
    z = m(x.as_subclass(Sub))
    assert Sub.seen and torch.equal(z.as_subclass(torch.Tensor), y)
