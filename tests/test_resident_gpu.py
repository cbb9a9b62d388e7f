"""GPU parity tests of the resident plan (csrc/gn_resident.cu): both passes in one cooperative kernel, one CTA
per SM, the last tiles of a CTA's row range kept in shared memory between the passes.

GNB200_RESIDENT_CTAS / _STAGES bound the grid and the ring, so that tile remainders, stage reuse in both
passes and ranges of one short tile are reached at sizes the CPU oracle finishes in seconds.
Tolerances as everywhere: 1e-5 (fp32), 1e-2 (fp16 / bf16), max-abs error relative to max(1, max|oracle|).
"""
import pytest
import torch

from oracle import gn_oracle as O

from .test_parity_gpu import DT, check_against, run_cabi

pytestmark = pytest.mark.gpu

CASES = [
    # (N, C, spatial, G, dtype, act, CTAs per sample, stages)
    (1, 256, (96, 96), 32, "float16", "silu", 0, 16),        # every SM, one or two tiles each, all resident
    (2, 256, (96, 97), 32, "bfloat16", "gelu", 5, 2),         # many tiles through two stages, ragged last tile
    (3, 128, (40, 57), 32, "float32", "gelu_tanh", 3, 3),     # fp32: Welford, xh form
    (2, 320, (33, 47), 32, "float16", "silu", 4, 3),          # D = 10: vectors straddle groups; 32 idle threads
    (1, 40, (131, 17), 8, "float32", "relu", 2, 2),           # D = 5, 10 vectors per row
    (1, 64, (57, 31), 64, "float32", "identity", 7, 2),       # D = 1
    (1, 2048, (9, 11), 32, "bfloat16", "silu", 3, 2),         # two row lanes
    (1, 4096, (5, 7), 1, "float16", "gelu_tanh", 2, 2),       # one row lane: the widest row
    (1, 8, (301, 3), 1, "float16", "identity", 2, 2),         # one vector per row
    (148, 64, (8, 8), 8, "float16", "silu", 0, 16),           # one CTA per sample
    (1, 128, (1, 5), 4, "float32", "silu", 0, 16),            # fewer rows than CTAs
]


@pytest.fixture(scope="module")
def nt():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from channels_last_groupnorm_b200 import _native

    return _native


@pytest.mark.parametrize("case", CASES, ids=lambda c: "%dx%dx%s-g%d-%s-%s-%d-%d" % (c[0], c[1], "x".join(map(str, c[2])), *c[3:]))
def test_resident_plan_against_oracle(nt, case, monkeypatch):
    N, C, sp, G, dt, act, ctas, stages = case
    monkeypatch.setenv("GNB200_FORCE_PATH", "resident")
    monkeypatch.setenv("GNB200_RESIDENT_CTAS", str(ctas))
    monkeypatch.setenv("GNB200_RESIDENT_STAGES", str(stages))
    for direction in (0, 1):
        assert " resident=1 " in nt.describe_plan(N, sp[0] * sp[1], C, G, DT[dt], direction)
    x, ga, be, dy = O.make_inputs(N, C, sp, DT[dt], seed=23, x_dist="uniform3")
    out = run_cabi(nt, x, ga, be, dy, G, 1e-5, act)
    want = O.oracle_c(x, ga, be, dy, G, 1e-5, act, threads=4)
    check_against(out, want, DT[dt])
    assert O.rel_err(out["mean"], want["mean"]) < 1e-5
    assert O.rel_err(out["rstd"] / want["rstd"].cuda().float(), torch.ones_like(want["rstd"])) < 1e-5
    assert O.rel_err(out["dparam"][0], want["dgamma"]) <= O.TOLERANCE[DT[dt]]
    assert O.rel_err(out["dparam"][1], want["dbeta"]) <= O.TOLERANCE[DT[dt]]
    again = run_cabi(nt, x, ga, be, dy, G, 1e-5, act)  # fixed summation order: bit-identical reruns
    for k in ("y", "dx", "dparam", "mean", "rstd"):
        assert torch.equal(out[k], again[k]), k
    assert nt.wait_timeouts() == 0


@pytest.mark.parametrize("dt", ["float16", "float32"])
@pytest.mark.parametrize("refused_by", [1, 2], ids=["check", "runtime"])
def test_a_grid_that_cannot_be_resident_takes_the_other_plan(nt, refused_by, dt, monkeypatch):
    """A device that this process shares may refuse the cooperative grid, in the occupancy check or at the launch itself.
    The call then runs the multi-kernel (or wave) plan and leaves no error behind."""
    from .test_parity_gpu import _flat

    N, C, sp, G, act = 1, 64, (65, 41), 8, O.ACT_CODES["silu"]
    x, ga, be, dy = O.make_inputs(N, C, sp, DT[dt], seed=29)
    want = O.oracle_c(x, ga, be, dy, G, 1e-5, "silu", threads=4)
    xd, dyd, gd, bd = _flat(x.cuda()), _flat(dy.cuda()), ga.cuda(), be.cuda()
    monkeypatch.setenv("GNB200_FORCE_PATH", "twopass")
    plain = nt.fwd_raw(xd, gd, bd, G, 1e-5, act)
    monkeypatch.setenv("GNB200_FORCE_PATH", "resident")
    nt.check(nt.lib.gnb200_debug_next_resident(refused_by, 0))
    y, mean, rstd = nt.fwd_raw(xd, gd, bd, G, 1e-5, act)
    assert torch.equal(y, plain[0]) and torch.equal(mean, plain[1]) and torch.equal(rstd, plain[2])
    nt.check(nt.lib.gnb200_debug_next_resident(refused_by, 0))
    dx, dparam, dgamma, dbeta = nt.bwd_raw(dyd, xd, gd, bd, mean, rstd, G, act)
    assert O.rel_err(dx.reshape(N, *sp, C).permute(0, 3, 1, 2), want["dx"]) <= O.TOLERANCE[DT[dt]]
    assert O.rel_err(dgamma, want["dgamma"]) <= O.TOLERANCE[DT[dt]] and O.rel_err(dbeta, want["dbeta"]) <= O.TOLERANCE[DT[dt]]
    assert torch.equal(xd + 1, 1 + xd)  # (a torch launch checks the last error)
    torch.cuda.synchronize()
    again = nt.fwd_raw(xd, gd, bd, G, 1e-5, act)  # the hook held for one launch: resident again
    assert O.rel_err(again[1], want["mean"]) < 1e-5


@pytest.mark.parametrize("what", [3, 4, 5], ids=["no arrival", "no first copy", "no copy of the second pass"])
@pytest.mark.parametrize("dt,act", [("float16", "relu"), ("float32", "silu")])
def test_waits_that_run_out_leave_nan_and_a_status(nt, what, dt, act, monkeypatch):
    """One CTA withholds what others, or its own threads, wait for (decided on the host, wait limit one millisecond).  The
    call returns, the outputs that depend on it are NaN - for ReLU too, which maps a NaN pre-activation to 0 - the rest is
    what it should be, the next call reports the failure, and after re-arming everything runs as before."""
    from .test_parity_gpu import _flat

    N, C, sp, G, code, ctas, cta = 2, 64, (32, 120), 8, O.ACT_CODES[act], 3, 1
    monkeypatch.setenv("GNB200_FORCE_PATH", "resident")
    monkeypatch.setenv("GNB200_RESIDENT_CTAS", str(ctas))
    monkeypatch.setenv("GNB200_RESIDENT_STAGES", "2")
    x, ga, be, dy = O.make_inputs(N, C, sp, DT[dt], seed=37)
    xd, dyd, gd, bd = _flat(x.cuda()), _flat(dy.cuda()), ga.cuda(), be.cuda()
    good = nt.fwd_raw(xd, gd, bd, G, 1e-5, code)
    mean, rstd = good[1], good[2]
    good_b = nt.bwd_raw(dyd, xd, gd, bd, mean, rstd, G, code)
    plans = [dict(kv.split("=") for kv in nt.describe_plan(N, sp[0] * sp[1], C, G, DT[dt], d).split()[2:]) for d in (0, 1)]

    def run(direction):
        nt.check(nt.lib.gnb200_debug_next_resident(what, cta))
        try:
            out = nt.fwd_raw(xd, gd, bd, G, 1e-5, code) if direction == 0 else nt.bwd_raw(dyd, xd, gd, bd, mean, rstd, G, code)
            torch.cuda.synchronize()  # the call returns and the GPU still answers
            assert nt.wait_timeouts() > 0
            with pytest.raises(nt.Gnb200Error) as err:
                nt.fwd_raw(xd, gd, bd, G, 1e-5, code)
            assert err.value.status == nt.ERR_EXCHANGE_TIMEOUT
        finally:
            nt.clear_wait_timeouts()
        return out

    for direction, want in ((0, good), (1, good_b)):
        got = run(direction)
        if what != 5:
            assert all(torch.isnan(t.float()).all() for t in got)
            continue
        # the CTA's rows: tiles of `tile` rows; the second pass takes them from the last to the first, two stages hold the
        # last two, so the third from the end is missing, with all before it
        rows, tile = int(plans[direction]["rows"]), int(plans[direction]["tile"].split("x")[1])
        tiles = -(-rows // tile)
        assert tiles >= 4
        missing = torch.zeros(sp[0] * sp[1], dtype=torch.bool, device="cuda")
        missing[cta * rows:cta * rows + (tiles - 2) * tile] = True
        assert torch.isnan(got[0][0, missing].float()).all()
        assert torch.equal(got[0][0, ~missing], want[0][0, ~missing]) and torch.equal(got[0][1], want[0][1])
        if direction == 0:
            assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
        else:  # parameter gradients: those that this CTA adds up
            lost = torch.isnan(got[1][0])
            assert lost.any() and torch.equal(got[1][:, ~lost], want[1][:, ~lost])
    assert nt.wait_timeouts() == 0
    again = nt.fwd_raw(xd, gd, bd, G, 1e-5, code)
    assert all(torch.equal(a, b) for a, b in zip(again, good))


def test_peer_entry_points_with_one_rank_after_the_resident_backward(nt, monkeypatch):
    """The exchange of the parameter gradients follows the resident kernel as it follows the wave kernel: with one rank
    the results are those of the plain call.  (Several ranks need one GPU each: tests/test_peer_multigpu.py, bench.py.)"""
    from .test_parity_gpu import _flat

    monkeypatch.setenv("GNB200_FORCE_PATH", "resident")
    N, C, sp, G, act = 2, 64, (40, 41), 8, O.ACT_CODES["gelu"]
    x, ga, be, dy = O.make_inputs(N, C, sp, torch.bfloat16, seed=41)
    xd, dyd, gd, bd = _flat(x.cuda()), _flat(dy.cuda()), ga.cuda(), be.cuda()
    _, mean, rstd = nt.fwd_raw(xd, gd, bd, G, 1e-5, act)
    want = nt.bwd_raw(dyd, xd, gd, bd, mean, rstd, G, act)
    buf = torch.zeros(nt.peer_exchange_bytes(C, 1) // 4, device="cuda")
    for collect in (True, False):
        dx, dparam = nt.bwd_peer_raw(dyd, xd, gd, bd, mean, rstd, G, act, [buf.data_ptr()], 0, collect=collect)
        assert torch.equal(dx, want[0]) and torch.equal(dparam, want[1])
    torch.cuda.synchronize()
    assert int(buf.abs().sum().item()) == 0 and nt.wait_timeouts() == 0


def test_resident_plan_in_a_captured_graph(nt):
    """Unforced, both directions: one memset node and one cooperative kernel each; replays see new inputs."""
    N, R, C, G = 1, 98304, 256, 8
    x, dy = (torch.randn(N, R, C, device="cuda", dtype=torch.float16) for _ in range(2))
    ga, be = torch.ones(C, device="cuda", dtype=torch.float16), torch.zeros(C, device="cuda", dtype=torch.float16)
    for d in (0, 1):
        assert " resident " in nt.describe_plan(N, R, C, G, torch.float16, d)

    def step():
        y, mean, rstd = nt.fwd_raw(x, ga, be, G, 1e-5, 2)
        return (y, mean, rstd) + nt.bwd_raw(dy, x, ga, be, mean, rstd, G, 2)

    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        step()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        out = step()
    x.mul_(0.5).add_(1.0)
    g.replay()
    g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(out, step())) and nt.wait_timeouts() == 0
