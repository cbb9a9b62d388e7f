"""Column blocks with more groups than the CTA has threads (csrc/gn_reduce.cuh): groups narrower than a vector, few rows."""
import pytest
import torch

from channels_last_groupnorm_b200 import _native as nt
from oracle import gn_oracle as O

DT = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}


def _plan(N, R, C, G, dtype):
    text = nt.describe_plan(N, R, C, G, dtype, 0)
    return text, {k: int(v) for k, v in (kv.split("=") for kv in text.split()[2:]) if v.isdigit()}


def test_only_groups_narrower_than_a_vector_outnumber_the_threads(monkeypatch):
    """crew_moments and crew_group_sums give a thread one group except in the branch for narrow groups: no plan may need more."""
    outnumbered = 0
    for force in (None, "resident"):
        if force:
            monkeypatch.setenv("GNB200_FORCE_PATH", force)
        for dtype, ve in ((torch.float16, 8), (torch.float32, 4)):
            for D in (1, 2, 3, 4, 5, 7, 8, 9, 10, 12, 16, 24, 30, 64):
                for C in (24, 40, 42, 96, 120, 128, 320, 640, 768, 1280, 2560, 4096):
                    if C % D:
                        continue
                    for R in (1, 4, 9, 25, 64, 300):
                        for N in (1, 8, 64, 300) if not force else (1, 8):
                            text, p = _plan(N, R, C, C // D, dtype)
                            if " twopass " in text:
                                continue
                            many = p["cw"] // D > p["threads"]
                            assert not many or (D < p["ve"] and " fused " in text), text
                            outnumbered += many
    assert outnumbered > 0


@pytest.mark.gpu
@pytest.mark.parametrize("N,R,C,G,dt", [
    (64, 1, 40, 40, "float16"),       # 32 threads, 40 groups of one element each
    (64, 4, 40, 40, "bfloat16"),      # a cluster of four
    (8, 36, 40, 40, "float16"),       # eight CTAs, five row lanes
    (300, 4, 320, 320, "float16"),    # 64 threads, 80 groups
    (64, 25, 1280, 1280, "float16"),  # 128 threads, 160 groups
    (300, 16, 640, 320, "bfloat16"),  # two channels per group
    (300, 16, 768, 256, "float16"),   # three: 96 threads, 128 groups
    (300, 36, 384, 128, "float16"),   # the same in a cluster of two
    (300, 16, 640, 128, "float16"),   # five
    (64, 9, 5120, 1024, "bfloat16"),
    (300, 16, 320, 320, "float32"),
    (64, 16, 1280, 640, "float32"),   # 160 groups, 96 threads
], ids=lambda v: str(v))
def test_more_groups_than_threads(N, R, C, G, dt):
    from .test_parity_gpu import check_against, run_cabi

    text, p = _plan(N, R, C, G, DT[dt])
    assert " fused " in text and p["cw"] * G // C > p["threads"], text
    x, ga, be, dy = O.make_inputs(N, C, (R, 1), DT[dt], seed=59, x_dist="uniform3")
    out = run_cabi(nt, x, ga, be, None, G, 1e-5, "silu")
    want = O.oracle_c(x, ga, be, dy, G, 1e-5, "silu", threads=4)
    check_against(out, want, DT[dt], keys=("y",))
    # fp32: a few units of 2^-24 in the mean; sums about a thread's first row can lose as many in the variance as there are rows
    assert O.rel_err(out["mean"], want["mean"]) < 1e-6
    assert O.rel_err(out["rstd"] / want["rstd"].cuda().float(), torch.ones_like(want["rstd"])) < 1e-5
    assert nt.wait_timeouts() == 0
