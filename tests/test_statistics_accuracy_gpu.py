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
    elif kind == "one huge":  # its square is just within fp32
        x[0, 0, 0] = 1e19 if x.dtype is torch.bfloat16 else 6e4
    elif kind == "offset 100":
        x += 100
    return x


@pytest.mark.parametrize("kind", ["normal", "first 60000", "offset 100", "one huge"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=lambda d: str(d)[6:])
@pytest.mark.parametrize("shape", [(1, 128, 1 << 20, 32), (4, 320, 9216, 32), (2, 24, 40, 3)], ids=str)
def test_channels_first_statistics(shape, dtype, kind):
    N, C, R, G = shape
    torch.manual_seed(1)
    x = torch.randn(N, C, R, device="cuda", dtype=dtype)
    _disturb(x.transpose(1, 2), kind)
    _check(x, G)


@pytest.mark.parametrize("kind", ["normal", "first 3000", "offset 100"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32], ids=lambda d: str(d)[6:])
@pytest.mark.parametrize("G", [32, 64], ids=lambda g: "g%d" % g)  # 16-bit: one shift for a vector's lanes / a shift per lane
def test_long_row_ranges_of_the_resident_forward(G, dtype, kind, monkeypatch):
    """Two CTAs for 262144 rows: 4096 rows per thread (fp32: 8192), as a sample of several GB has.  They are
    summed in pieces of n = 32; next to an outlier that is the shift of a piece, M2 may be off by n^1.5 u = 181 u, rstd
    by half of that, and twice as much is allowed."""
    monkeypatch.setenv("GNB200_FORCE_PATH", "resident")
    monkeypatch.setenv("GNB200_RESIDENT_CTAS", "2")
    torch.manual_seed(1)
    x = torch.randn(1, 1 << 18, 128, device="cuda", dtype=dtype)
    _check(_disturb(x, kind).permute(0, 2, 1), G, bound=1.1e-5 if kind == "first 3000" and dtype is not torch.float32 else RSTD)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32], ids=lambda d: str(d)[6:])
def test_long_row_ranges_of_the_resident_backward(dtype, monkeypatch):
    """dgamma of x around 100 with mean = 100 and rstd = 1 (exact, so that only the sums round).  A piece of 32 rows
    adds up to 3200, each step rounds by 2^-13 at most: about 32^0.5 * 2^-14 per piece and 8192^0.5 times that over the
    pieces, 0.03; the tree above adds numbers of up to 100 * 2^18 / 64 with an error of 2^-6 each, 64^0.5 times that: 0.13.  Twice the sum
    is allowed (sums over a thread's whole range: 9).  dbeta, 2^18, may be off by eight u."""
    monkeypatch.setenv("GNB200_FORCE_PATH", "resident")
    monkeypatch.setenv("GNB200_RESIDENT_CTAS", "2")
    import channels_last_groupnorm_b200  # noqa: F401

    torch.manual_seed(2)
    N, R, C, G = 1, 1 << 18, 128, 32
    x = (torch.randn(N, R, C, device="cuda") + 100).to(dtype).permute(0, 2, 1)
    dy = (torch.rand(N, R, C, device="cuda") + 0.5).to(dtype).permute(0, 2, 1)
    one = torch.ones(C, device="cuda", dtype=dtype)
    mean, rstd = torch.full((N, G), 100.0, device="cuda"), torch.ones(N, G, device="cuda")
    _, dparam = torch.ops.gnb200.bwd_f32(dy, x, one, one, mean, rstd, G, 0)
    want = (dy.double() * (x.double() - 100)).sum((0, 2)), dy.double().sum((0, 2))
    off = (dparam[0] - want[0]).abs().max().item(), (dparam[1] - want[1]).abs().max().item()
    assert off[0] <= 0.32 and off[1] <= 0.125, off
