"""The rule that takes a slab which fits a cluster to a multi-pass plan all the same (gn_plan.cu, fused_loses): both sides of
its lines, what a caller with the fused plan's scratch gets, and the results on either path."""
import pytest
import torch

from channels_last_groupnorm_b200 import _native as nt
from oracle import gn_oracle as O

F16, BF16, F32 = torch.float16, torch.bfloat16, torch.float32
NAME = {0: "fwd", 1: "bwd"}


def _fused(shape, dtype, direction):
    return nt.describe_plan(*shape, dtype, direction).startswith("%s fused " % NAME[direction])


@pytest.mark.parametrize("shape,dtype,fused", [
    ((1, 65536, 256, 32), F16, False),    # 16-byte segments, one CTA per SM
    ((2, 40000, 256, 32), BF16, False),   # 32-byte segments
    ((1, 28700, 512, 32), F16, False),    # 64-byte segments: the widest
    ((1, 40000, 256, 32), F32, False),
    ((1, 65536, 16, 4), F16, False),      # 2.1 MB ...
    ((1, 40000, 24, 6), BF16, True),      # ... and 1.9
    ((4, 7744, 2560, 32), F16, True),     # 160-byte segments
    ((13, 18632, 40, 8), BF16, True),     # whole rows of 80 bytes
    ((1, 16384, 512, 32), F16, True),     # 32-byte segments, several CTAs per SM
    ((12, 25745, 12, 1), F32, True),      # whole rows
    ((64, 4096, 256, 32), BF16, True),
], ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v).replace("torch.", ""))
def test_which_calls_leave_the_fused_plan(shape, dtype, fused, monkeypatch):
    for direction in (0, 1):
        text = nt.describe_plan(*shape, dtype, direction)
        assert _fused(shape, dtype, direction) is fused, text
        query = nt.lib.gnb200_fwd_workspace_bytes if direction == 0 else nt.lib.gnb200_bwd_workspace_bytes
        assert int(dict(kv.split("=") for kv in text.split()[2:])["ws"]) <= query(*shape, nt.DTYPE_CODES[dtype])
    monkeypatch.setenv("GNB200_FORCE_PATH", "fused")
    assert all(_fused(shape, dtype, d) for d in (0, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("shape,dtype,act", [((1, 50021, 64, 8), F16, "silu"), ((1, 65537, 32, 8), BF16, "gelu"), ((1, 40000, 64, 16), F32, "gelu_tanh")],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v).replace("torch.", ""))
def test_callers_with_little_scratch_get_the_fused_plan(shape, dtype, act, monkeypatch):
    """Without scratch (forward), with the fused plan's (backward) and with the library's own array the calls run as they did
    before there was the rule, bit for bit; with what the queries ask for they are as exact."""
    N, R, C, G = shape
    code, dt = O.ACT_CODES[act], nt.DTYPE_CODES[dtype]
    x, ga, be, dy = O.make_inputs(N, C, (R, 1), dtype, seed=47)
    want = O.oracle_c(x, ga, be, dy, G, 1e-5, act, threads=4)
    xd, dyd = (t.cuda().permute(0, 2, 3, 1).reshape(N, R, C).contiguous() for t in (x, dy))
    gd, bd = ga.cuda(), be.cuda()
    usual = nt.fwd_raw(xd, gd, bd, G, 1e-5, code)
    usual_b = nt.bwd_raw(dyd, xd, gd, bd, usual[1], usual[2], G, code)
    assert not any(_fused(shape, dtype, d) for d in (0, 1))
    s = torch.cuda.current_stream().cuda_stream
    y, mean, rstd = torch.empty_like(xd), torch.empty(N, G, device="cuda"), torch.empty(N, G, device="cuda")
    p = lambda t: t.data_ptr()
    nt.check(nt.lib.gnb200_fwd(p(xd), p(gd), p(bd), N, R, C, G, 1e-5, code, dt, p(y), p(mean), p(rstd), None, 0, s))
    dx, dparam = torch.empty_like(xd), torch.empty(2, C, device="cuda")
    dg, db = torch.empty_like(gd), torch.empty_like(gd)
    monkeypatch.setenv("GNB200_FORCE_PATH", "fused")
    fused = nt.fwd_raw(xd, gd, bd, G, 1e-5, code)
    fused_b = nt.bwd_raw(dyd, xd, gd, bd, usual[1], usual[2], G, code)
    need = nt.lib.gnb200_bwd_workspace_bytes(N, R, C, G, dt)
    monkeypatch.delenv("GNB200_FORCE_PATH")
    assert all(torch.equal(a, b) for a, b in zip((y, mean, rstd), fused))
    ws = torch.empty(need, device="cuda", dtype=torch.uint8)
    nt.check(nt.lib.gnb200_bwd(p(dyd), p(xd), p(gd), p(bd), p(usual[1]), p(usual[2]), N, R, C, G, code, dt, p(dx), p(dparam), p(dg),
                               p(db), p(ws), need, s))
    assert all(torch.equal(a, b) for a, b in zip((dx, dparam, dg, db), fused_b))
    nt.bwd_static_scratch_raw(dyd, xd, gd, bd, usual[1], usual[2], G, code, dx, dparam, dg, db)
    for got in ((usual[0], usual_b[0], usual_b[1]), (y, dx, dparam)):
        for t, k in zip(got[:2], ("y", "dx")):
            assert O.rel_err(t.reshape(N, R, 1, C).permute(0, 3, 1, 2), want[k]) <= O.TOLERANCE[dtype]
        assert O.rel_err(got[2][0], want["dgamma"]) <= O.TOLERANCE[dtype] and O.rel_err(got[2][1], want["dbeta"]) <= O.TOLERANCE[dtype]
