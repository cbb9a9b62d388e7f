"""Every plan that stands in for a fused one fits an SM's shared memory: many narrow groups (gn_plan.cu, make_plan_inner)."""
import pytest
import torch

from channels_last_groupnorm_b200 import _native as nt
from oracle import gn_oracle as O

F16, BF16, F32 = torch.float16, torch.bfloat16, torch.float32
SMEM = 227 * 1024


def test_calls_that_a_fused_plan_can_take_have_a_plan_that_fits(monkeypatch):
    left = 0
    for dtype in (F16, F32):
        for C in (64, 320, 768, 1024, 1280, 2048, 2560, 5120):
            for D in (1, 2, 3, 5, 8, 64):
                if C % D:
                    continue
                for R in (12000, 18000, 28700, 50000, 100000):
                    for N in (1, 3):
                        for direction in (0, 1):
                            text = nt.describe_plan(N, R, C, C // D, dtype, direction)
                            smem = int(dict(kv.split("=") for kv in text.split()[2:])["smem"])
                            if smem > SMEM:
                                monkeypatch.setenv("GNB200_FORCE_PATH", "fused")
                                assert " fused " not in nt.describe_plan(N, R, C, C // D, dtype, direction), text
                                monkeypatch.delenv("GNB200_FORCE_PATH")
                            left += " fused " not in text
    assert left > 0


@pytest.mark.gpu
@pytest.mark.parametrize("N,R,C,G,dt", [(1, 18000, 1024, 1024, F16), (1, 14500, 2048, 1024, BF16), (1, 14500, 1024, 1024, F32)],
                         ids=lambda v: str(v).replace("torch.", ""))
def test_many_narrow_groups_of_many_rows(N, R, C, G, dt):
    from .test_parity_gpu import check_against, run_cabi

    x, ga, be, dy = O.make_inputs(N, C, (R, 1), dt, seed=61, x_dist="uniform3")
    out = run_cabi(nt, x, ga, be, dy, G, 1e-5, "silu")
    check_against(out, O.oracle_c(x, ga, be, dy, G, 1e-5, "silu", threads=4), dt)
