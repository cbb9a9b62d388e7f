"""What the module's autograd node saves: the input as a flat (N, C, R) tensor of its own over the same storage, whichever way
the call takes, so that what looks at or replaces saved tensors meets the same on both."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

import channels_last_groupnorm_b200 as pkg

pytestmark = pytest.mark.gpu


class Pass(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def _input(order, shape=(2, 32, 6, 5), dtype=torch.float32):
    t = torch.randn(shape, device="cuda", dtype=dtype)
    return t.to(memory_format=torch.channels_last) if order == "last" else t


def _grads(y, m, x):
    return torch.autograd.grad(y.square().sum(), (x, m.weight, m.bias))


def _equal(got, want):
    return all(torch.equal(a, b) and a.stride() == b.stride() for a, b in zip(got, want))


@pytest.mark.parametrize("order", ["last", "first"])
@pytest.mark.parametrize("shape", [(2, 32, 6, 5), (3, 16, 7), (2, 8, 1, 1), (1, 8, 1, 6), (2, 1, 4, 4)], ids=lambda s: "x".join(map(str, s)))
def test_hooks_are_given_the_same_on_both_paths(order, shape):
    torch.manual_seed(5)
    m = pkg.GN_NHWC(min(4, shape[1]), shape[1], activation="silu", device="cuda")
    x = (_input(order, shape) if len(shape) == 4 else torch.randn(shape, device="cuda")).requires_grad_(True)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t) or t, lambda t: t):
        y = m(x)
        with Pass():
            want = m(x)
    assert len(seen) == 10
    for a, b in zip(seen[:5], seen[5:]):
        assert a.shape == b.shape and a.dtype == b.dtype
        assert a.shape.numel() == 1 or [s for s, n in zip(a.stride(), a.shape) if n > 1] == [s for s, n in zip(b.stride(), b.shape) if n > 1]
    assert seen[0].data_ptr() == seen[5].data_ptr() == x.data_ptr()
    assert _equal(_grads(y, m, x), _grads(want, m, x))


@pytest.mark.parametrize("order", ["last", "first"])
def test_checkpoint_that_is_recomputed_under_a_profiler(order):
    """Forward without, recomputation with a profiler: the second takes the general path, and must save the same kind of tensors."""
    from torch.utils.checkpoint import checkpoint

    m = pkg.GN_NHWC(4, 32, activation="gelu", device="cuda")
    x = _input(order).requires_grad_(True)
    want = _grads(m(x), m, x)
    y = checkpoint(m, x, use_reentrant=False)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]):
        got = _grads(y, m, x)
    assert _equal(got, want)
    with Pass():
        y = checkpoint(m, x, use_reentrant=False)
    assert _equal(_grads(y, m, x), want)


@pytest.mark.parametrize("needs", [True, False], ids=["leaf", "frozen"])
@pytest.mark.parametrize("order", ["last", "first"])
def test_input_whose_data_is_replaced_before_the_backward(order, needs):
    """`x.data = ...` gives the tensor object another storage; the node keeps the one that it has seen."""
    m = pkg.GN_NHWC(4, 32, activation="silu", device="cuda")
    x = _input(order).requires_grad_(needs)
    inputs = ((x,) if needs else ()) + (m.weight, m.bias)
    want = torch.autograd.grad(m(x).square().sum(), inputs)
    y = m(x)
    x.data = _input(order)
    assert _equal(torch.autograd.grad(y.square().sum(), inputs), want)


@pytest.mark.parametrize("pin", [False, True], ids=["pageable", "pinned"])
@pytest.mark.parametrize("order", ["last", "first"])
def test_saved_on_the_cpu(order, pin):
    """The pinned copies come back contiguous, in another storage order than they had."""
    m = pkg.GN_NHWC(4, 32, activation="silu", device="cuda", dtype=torch.float16)
    x = _input(order, dtype=torch.float16).requires_grad_(True)
    want = _grads(m(x).float(), m, x)
    for general in (False, True):
        with torch.autograd.graph.save_on_cpu(pin_memory=pin):
            if general:
                with Pass():
                    y = m(x)
            else:
                y = m(x)
        assert _equal(_grads(y.float(), m, x), want)
