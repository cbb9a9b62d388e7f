"""The module's native autograd node (torch.ops.gnb200.group_norm_act) against GN_NHWC_Func, which it stands in
for: same ops on the same views, so results and gradients are equal bit for bit, for every layout, rank, dtype and
parameter dtype that the module takes, and what lies beside a plain call (hooks, transforms, modes) behaves alike."""
import pytest
import torch

import channels_last_groupnorm_b200 as pkg

pytestmark = pytest.mark.gpu


def _tensor(shape, order, dtype):
    t = torch.randn(shape, device="cuda", dtype=dtype)
    if order == "last":
        nd = t.ndim
        t = t.permute(0, *range(2, nd), 1).contiguous().permute(0, nd - 1, *range(1, nd - 1))
    elif order == "sliced":  # unit channel stride, but rows with a gap
        t = torch.randn((shape[0], *shape[2:], 2 * shape[1]), device="cuda", dtype=dtype)[..., :shape[1]]
        t = t.permute(0, t.ndim - 1, *range(1, t.ndim - 1))
    return t


CASES = [
    ((2, 32, 5, 7), "last", torch.float16, torch.float16),
    ((2, 32, 5, 7), "first", torch.bfloat16, torch.float32),
    ((1, 24, 9, 3), "sliced", torch.float32, torch.float32),
    ((3, 16, 11), "last", torch.bfloat16, torch.bfloat16),
    ((2, 8, 3, 4, 5), "last", torch.float16, torch.float32),
    ((2, 8, 3, 4, 5), "first", torch.float64, torch.float64),
    ((2, 8, 1, 1), "first", torch.float32, torch.float32),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "%s-%s-%s-%s" % ("x".join(map(str, c[0])), c[1], str(c[2])[6:], str(c[3])[6:]))
@pytest.mark.parametrize("dy_order", ["last", "first"])
def test_native_node_equals_the_python_function(case, dy_order):
    shape, order, dtype, pdtype = case
    torch.manual_seed(7)
    m = pkg.GN_NHWC(4, shape[1], activation="silu", device="cuda", dtype=pdtype)
    x = _tensor(shape, order, dtype).requires_grad_(True)
    dy = _tensor(shape, dy_order, dtype)
    got = m(x)
    want = pkg.GN_NHWC_Func.apply(x, m.weight, m.bias, 4, m.eps, m.act_code)
    assert "GnFunction" in got.grad_fn.name() and got.stride() == want.stride() and torch.equal(got, want)
    inputs = (x, m.weight, m.bias)
    for a, b, p in zip(torch.autograd.grad(got, inputs, dy), torch.autograd.grad(want, inputs, dy), inputs):
        assert a.dtype == b.dtype == p.dtype and a.stride() == b.stride() and torch.equal(a, b)
    with torch.no_grad():
        assert torch.equal(m(x), want)
    with torch.inference_mode():
        assert torch.equal(m(x), want)


def test_what_surrounds_a_call_behaves_as_with_the_python_function():
    m = pkg.GN_NHWC(4, 32, activation="gelu", device="cuda")
    x = _tensor((2, 32, 6, 6), "last", torch.float32).requires_grad_(True)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or len(packed) - 1, lambda i: packed[i]):
        y = m(x)
    assert len(packed) == 5
    y.sum().backward()
    from torch.utils.checkpoint import checkpoint

    x2 = x.detach().requires_grad_(True)
    checkpoint(m, x2, use_reentrant=False).sum().backward()
    assert torch.equal(x.grad, x2.grad)
    y = m(x)  # the saved input changed: refused
    with torch.no_grad():
        x.add_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()
    with torch.autograd.forward_ad.dual_level():  # no forward-mode formula
        dual = torch.autograd.forward_ad.make_dual(x.detach(), torch.ones_like(x))
        with pytest.raises(RuntimeError):
            m(dual)
    with pytest.raises(RuntimeError):  # no vmap rule
        torch.vmap(m)(torch.randn(2, 2, 32, 4, 4, device="cuda"))
    from torch.utils._python_dispatch import TorchDispatchMode

    seen = []

    class Record(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    with Record():
        m(x).sum().backward()
    assert any("gnb200.fwd" in s for s in seen) and any("gnb200.bwd" in s for s in seen)


def test_cuda_graph_capture_of_a_training_step():
    m = pkg.GN_NHWC(8, 64, activation="silu", device="cuda", dtype=torch.float16)
    x = _tensor((2, 64, 16, 16), "last", torch.float16).requires_grad_(True)
    dy = _tensor((2, 64, 16, 16), "last", torch.float16)

    def step():
        return torch.autograd.grad(m(x), (x, m.weight, m.bias), dy)

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        step()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        out = step()
    with torch.no_grad():
        x.mul_(0.5)
    g.replay()
    torch.cuda.synchronize()
    for a, b in zip(out, step()):
        assert torch.equal(a, b)


@pytest.mark.parametrize("pdtype", [torch.float16, torch.float32], ids=["typed", "fp32-params"])
@pytest.mark.parametrize("order", ["last", "first"])
def test_compiled_autograd_traces_the_backward(order, pdtype):
    """As it does with a Python function: the node is part of the captured graph, not a call back into eager mode, and the
    gradients are those of the plain engine, also when a second input has another size."""
    from torch._dynamo import compiled_autograd

    m = pkg.GN_NHWC(4, 32, activation="silu", device="cuda", dtype=pdtype)
    graphs = []

    def run(x):
        m.zero_grad()
        x = x.clone().requires_grad_(True)
        (m(x) ** 2).sum().backward()
        return [x.grad] + [p.grad.clone() for p in m.parameters()]

    def capture(gm):
        graphs.append(" ".join(str(n.target) for n in gm.graph.nodes))
        return gm

    for shape in ((2, 32, 6, 6), (3, 32, 5, 7)):
        x = _tensor(shape, order, torch.float16)
        want = run(x)
        for compiler in (capture, torch.compile(backend="aot_eager")):
            with compiled_autograd._enable(compiler, dynamic=False):
                got = run(x)
            assert all(torch.equal(a, b) and a.stride() == b.stride() for a, b in zip(got, want))
    assert graphs and all("GnFunction" in g and "non_traceable" not in g for g in graphs)


def test_num_groups_and_eps_are_converted_as_before():
    """num_groups from a division and eps as text (a value read from a configuration file) are what int() and float()
    make of them."""
    x = _tensor((2, 32, 6, 6), "last", torch.float32)
    m = pkg.GN_NHWC(32 / 8, 32, eps="1e-5", device="cuda")
    assert torch.equal(m(x), pkg.GN_NHWC_Func.apply(x, m.weight, m.bias, 32 / 8, "1e-5", 0))
    assert torch.equal(m(x), pkg.GN_NHWC(4, 32, eps=1e-5, device="cuda")(x))
