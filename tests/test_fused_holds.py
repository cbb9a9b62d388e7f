"""Calls that keep the fused plan although it has one CTA per SM and narrow row segments (gn_plan.cu, fused_holds): shapes on both
sides of each line, with the times there; and the results."""
import pytest
import torch

from channels_last_groupnorm_b200 import _native as nt
from oracle import gn_oracle as O

F16, BF16, F32 = torch.float16, torch.bfloat16, torch.float32


def _path(shape, dtype, direction):
    return nt.describe_plan(*shape, dtype, direction).split()[1]


@pytest.mark.parametrize("shape,dtype,direction,path", [
    # backward, wave: units of a wave that do not fit one round
    ((77, 12838, 64, 32), BF16, 1, "fused"), ((58, 18448, 128, 16), F16, 1, "fused"), ((102, 14891, 64, 8), F32, 1, "fused"),
    ((8, 23864, 128, 32), F32, 1, "fused"), ((8, 25013, 128, 32), F32, 1, "wave"), ((16, 32598, 128, 32), F32, 1, "wave"),
    # ... groups of fewer than four channels; 64-byte segments in 512 threads; 128 threads; 16-byte segments
    ((10, 39733, 256, 256), F16, 1, "fused"), ((2, 50091, 256, 256), F32, 1, "fused"), ((2, 43811, 512, 64), F32, 1, "wave"),
    ((2, 12164, 512, 64), F32, 1, "fused"), ((13, 18857, 256, 64), F32, 1, "fused"), ((6, 13377, 512, 32), F32, 1, "wave"),
    ((4, 26755, 512, 32), F32, 1, "wave"), ((1, 52126, 256, 256), F32, 1, "wave"), ((7, 96947, 256, 256), F16, 1, "wave"),
    # forward, more than 128 groups
    ((1, 16441, 2048, 256), BF16, 0, "fused"), ((2, 25145, 512, 256), F32, 0, "fused"), ((5, 39536, 256, 128), F32, 0, "twopass"),
    ((1, 97326, 2048, 256), F16, 0, "twopass"),
    ((31, 12681, 128, 128), BF16, 0, "fused"),
    # clusters resident at once, short tiles
    ((3, 13570, 64, 4), F32, 1, "fused"), ((1, 40000, 64, 16), F32, 1, "wave"), ((1, 46536, 32, 4), F32, 1, "wave"), ((1, 23599, 96, 16), F32, 0, "twopass"),
    ((3, 17880, 128, 4), BF16, 0, "fused"), ((3, 17880, 128, 4), BF16, 1, "fused"),
    ((3, 29154, 48, 6), F16, 0, "fused"), ((3, 29154, 48, 6), F16, 1, "fused"),
    ((1, 57399, 128, 8), BF16, 0, "twopass"), ((1, 33402, 64, 16), F16, 0, "twopass"), ((1, 33402, 64, 16), F16, 1, "resident"),
    ((4, 28319, 192, 6), F16, 0, "twopass"), ((1, 25221, 192, 32), BF16, 1, "resident"),
    ((3, 46389, 64, 64), BF16, 0, "fused"), ((3, 46389, 64, 64), BF16, 1, "resident"),
], ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v).replace("torch.", ""))
def test_both_sides_of_the_lines(shape, dtype, direction, path, monkeypatch):
    assert _path(shape, dtype, direction) == path, nt.describe_plan(*shape, dtype, direction)
    monkeypatch.setenv("GNB200_FORCE_PATH", "fused")
    assert _path(shape, dtype, direction) == "fused"
    monkeypatch.setenv("GNB200_FORCE_PATH", "streaming")
    assert _path(shape, dtype, direction) != "fused"


@pytest.mark.gpu
@pytest.mark.parametrize("shape,dtype,act", [((3, 17880, 128, 4), BF16, "silu"), ((3, 29154, 48, 6), F16, "gelu"), ((3, 15172, 32, 16), F32, "gelu_tanh"),
                                             ((1, 13001, 256, 256), F32, "silu"), ((1, 8221, 1024, 256), F16, "identity")],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v).replace("torch.", ""))
def test_results(shape, dtype, act):
    from .test_parity_gpu import check_against, run_cabi

    N, R, C, G = shape
    x, ga, be, dy = O.make_inputs(N, C, (R, 1), dtype, seed=67)
    out = run_cabi(nt, x, ga, be, dy, G, 1e-5, act)
    check_against(out, O.oracle_c(x, ga, be, dy, G, 1e-5, act, threads=4), dtype)


@pytest.mark.parametrize("shape,dtype,threads", [((1, 22270, 640, 32), F32, 512), ((21, 18501, 24, 2), F32, 512), ((4, 7396, 240, 8), F16, 256)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v).replace("torch.", ""))
def test_scratch_of_the_reductions_leaves_room_for_the_larger_cta(shape, dtype, threads):
    """A few hundred bytes more than the reductions need had halved the CTA: 64 -> 70 us, 35 -> 49."""
    text = nt.describe_plan(*shape, dtype, 0)
    assert " fused " in text and int(dict(kv.split("=") for kv in text.split()[2:])["threads"]) == threads, text
