"""GPU tests that a group with an infinity or a NaN leaves the other groups alone: their outputs are the same bits as without it.
Vectors that straddle two groups are where they could mix (csrc/gn_reduce.cuh), in every plan that reduces them."""
import pytest
import torch

from oracle import gn_oracle as O

from .test_parity_gpu import DT, run_cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["auto", "resident", "twopass", "wave"])
@pytest.mark.parametrize("N,C,sp,G,dt", [
    (2, 320, (13, 11), 32, "float16"),   # D = 10, as in a U-Net
    (2, 240, (9, 17), 8, "bfloat16"),    # D = 30
    (2, 72, (13, 7), 8, "float16"),      # D = 9: parts of 1 .. 8 lanes
    (2, 40, (17, 9), 8, "float32"),      # D = 5 in fp32
    (2, 96, (7, 13), 32, "bfloat16"),    # D = 3, narrower than a vector
    (2, 128, (11, 13), 16, "float16"),   # D = 8: a vector per group
    (2, 42, (5, 9), 6, "float16"),       # D = 7 without vectors
], ids=lambda v: str(v).replace(" ", ""))
def test_the_other_groups_keep_their_bits(N, C, sp, G, dt, path, monkeypatch):
    from channels_last_groupnorm_b200 import _native as nt

    if path != "auto":
        monkeypatch.setenv("GNB200_FORCE_PATH", path)
    D = C // G
    x, ga, be, dy = O.make_inputs(N, C, sp, DT[dt], seed=53)
    want = run_cabi(nt, x, ga, be, dy, G, 1e-5, "silu")
    for group, channel, bad in ((0, D - 1, "inf"), (G // 2, 0, "nan"), (G // 2, D - 1, "-inf"), (G - 1, 0, "inf")):
        broken = x.clone()
        broken[1, group * D + channel, 2, 3] = float(bad)
        got = run_cabi(nt, broken, ga, be, dy, G, 1e-5, "silu")
        groups = torch.ones(N, G, dtype=torch.bool)
        groups[1, group] = False
        channels = groups.repeat_interleave(D, 1).cuda()
        groups = groups.cuda()
        assert not torch.isfinite(got["mean"][1, group])
        for k in ("mean", "rstd"):
            assert torch.equal(got[k][groups], want[k][groups]), (k, group, bad)
        for k in ("y", "dx"):
            assert torch.equal(got[k][channels], want[k][channels]), (k, group, bad)
        for k in ("dgamma", "dbeta"):
            assert torch.equal(got[k][channels[1]], want[k][channels[1]]), (k, group, bad)
