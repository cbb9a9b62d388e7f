"""GPU tests of the group moments of the fused forward plan (csrc/gn_reduce.cuh) where vectors straddle groups or groups are no
power of two of vectors: every width of the parts of a vector, row remainders, statistics against the fp64 oracle."""
import pytest
import torch

from oracle import gn_oracle as O

from .test_parity_gpu import DT, check_against, run_cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,C,sp,G,dt", [
    (1, 72, (13, 7), 8, "float16"),     # D = 9: parts of 1 .. 8 lanes
    (2, 200, (31, 9), 8, "bfloat16"),   # D = 25
    (1, 120, (17, 19), 8, "float16"),   # D = 15
    (2, 960, (16, 15), 32, "float16"),  # D = 30, as in the wider levels of a U-Net
    (1, 320, (37, 41), 32, "bfloat16"),  # D = 10, ragged rows over the cluster
    (1, 264, (23, 5), 11, "float16"),   # D = 24: three vectors per group
    (3, 96, (9, 11), 12, "float32"),    # D = 8 in fp32: two vectors per group
    (1, 60, (21, 13), 12, "float32"),   # D = 5 in fp32: parts of 1 .. 4 lanes
    (1, 56, (19, 3), 8, "bfloat16"),    # D = 7, narrower than a vector
    (5, 40, (1, 1), 4, "float16"),      # one pixel per sample
], ids=lambda v: str(v).replace(" ", ""))
@pytest.mark.parametrize("threads", [0, 512])
def test_statistics_of_straddling_groups(N, C, sp, G, dt, threads, monkeypatch):
    from channels_last_groupnorm_b200 import _native as nt

    if threads:
        monkeypatch.setenv("GNB200_THREADS", str(threads))
    assert " fused " in nt.describe_plan(N, sp[0] * sp[1], C, G, DT[dt], 0)
    x, ga, be, dy = O.make_inputs(N, C, sp, DT[dt], seed=43, x_dist="uniform3")
    x = (x.float() + 4.0 * torch.arange(C).remainder(5).view(1, C, *([1] * len(sp)))).to(DT[dt])  # channels of a group differ
    out = run_cabi(nt, x, ga, be, dy, G, 1e-5, "silu")
    want = O.oracle_c(x, ga, be, dy, G, 1e-5, "silu", threads=4)
    check_against(out, want, DT[dt])
    # fp32 sums of a few thousand values, two-pass: a few units of 2^-24
    assert O.rel_err(out["mean"], want["mean"]) < 1e-6
    assert O.rel_err(out["rstd"] / want["rstd"].cuda().float(), torch.ones_like(want["rstd"])) < 2e-6
