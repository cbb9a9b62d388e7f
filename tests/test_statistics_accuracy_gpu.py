"""Accuracy of mean and rstd against fp64 where a lossy way of summing shows: one element far from all others at the
place where a thread starts, a large common offset, and long runs per thread.

Bound: the sums are fp32 (unit roundoff u = 6e-8).  A thread, and the reductions after it, add a few dozen terms one
after the other and everything else in trees, so M2 is off by some ten u and rstd, its root, by half of that: 6e-7.  A
method that subtracts two numbers n times as large as M2 is off by n u instead, one that overflows by everything.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

RSTD = 6e-7


def _check(x, G, eps=1e-5, bound=RSTD):
    """x: (N, C, R) view in the layout under test."""
    import channels_last_groupnorm_b200  # noqa: F401

    N, C, R = x.shape
    one, zero = torch.ones(C, device="cuda", dtype=x.dtype), torch.zeros(C, device="cuda", dtype=x.dtype)
    _, mean, rstd = torch.ops.gnb200.fwd(x, one, zero, G, eps, 0)
    d = x.double().reshape(N, G, -1) if x.stride(2) == 1 else x.permute(0, 2, 1).double().reshape(N, R, G, -1).transpose(1, 2).reshape(N, G, -1)
    var, mu = torch.var_mean(d, -1, correction=0)
    want = (var + eps).rsqrt()
    off = ((rstd - want) / want).abs().max().item()
    assert off <= bound, off
    assert ((mean - mu) * want).abs().max().item() <= 2e-5  # (offset 100: 1700 u of the mean itself)


def _disturb(x, kind):
    """x: (N, positions, ...): the first positions are where the threads start."""
    if kind == "first 60000":
        x[:, 0] = 60000.0
    elif kind == "first 3000":
        x[:, 0] = 3000.0
    elif kind == "one 1e19":
        x[0, 0, 0] = 1e19
    elif kind == "offset 100":
        x += 100
    return x


@pytest.mark.parametrize("kind", ["normal", "first 60000", "offset 100", "one 1e19"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=lambda d: str(d)[6:])
@pytest.mark.parametrize("shape", [(1, 128, 1 << 20, 32), (4, 320, 9216, 32), (2, 24, 40, 3)], ids=str)
def test_channels_first_statistics(shape, dtype, kind):
    if kind == "one 1e19" and dtype is torch.float16:
        pytest.skip("beyond fp16")
    N, C, R, G = shape
    torch.manual_seed(1)
    x = torch.randn(N, C, R, device="cuda", dtype=dtype)
    _disturb(x.transpose(1, 2), kind)
    _check(x, G)
