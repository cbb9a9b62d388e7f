"""GPU tests of the tiles that the resident plan keeps in tensor memory (csrc/gn_resident.cu): where a tile waits between
the passes must not change a bit, whatever its row remainder, the number of stages or the number of parked tiles."""
import pytest
import torch

from oracle import gn_oracle as O

from .test_parity_gpu import DT, check_against, run_cabi

pytestmark = pytest.mark.gpu

CASES = [
    # (N, C, spatial, G, dtype, act, CTAs per sample): tiles of 128 / 64 rows at C = 128 (fp16) and so on
    (1, 128, (128, 9), 32, "float16", "silu", 1),       # forward: 9 tiles of 128 rows, backward: 18 of 64
    (1, 128, (1281, 1), 32, "bfloat16", "gelu", 1),     # one row beyond a whole tile
    (2, 320, (33, 47), 32, "float16", "silu", 3),       # D = 10; 480 of 512 threads, fifteen warps
    (1, 128, (40, 57), 32, "float32", "gelu_tanh", 3),  # fp32
    (1, 4096, (7, 11), 1, "float16", "relu", 1),        # one row lane
    (1, 1536, (61, 1), 4, "bfloat16", "identity", 1),   # two row lanes of 192 threads: twelve warps
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "%dx%dx%s-g%d-%s-%s-%d" % (c[0], c[1], "x".join(map(str, c[2])), *c[3:]))
def test_parked_tiles_change_no_bit(case, monkeypatch):
    from channels_last_groupnorm_b200 import _native as nt

    N, C, sp, G, dt, act, ctas = case
    monkeypatch.setenv("GNB200_FORCE_PATH", "resident")
    monkeypatch.setenv("GNB200_RESIDENT_CTAS", str(ctas))
    x, ga, be, dy = O.make_inputs(N, C, sp, DT[dt], seed=5, x_dist="uniform3")
    want = None
    for stages, park in ((2, 0), (2, 1), (2, 8), (3, 7), (5, 4), (16, 8)):
        monkeypatch.setenv("GNB200_RESIDENT_STAGES", str(stages))
        monkeypatch.setenv("GNB200_RESIDENT_PARK", str(park))
        out = run_cabi(nt, x, ga, be, dy, G, 1e-5, act)
        if want is None:
            want = out
            check_against(out, O.oracle_c(x, ga, be, dy, G, 1e-5, act, threads=4), DT[dt])
        for k in ("y", "dx", "dparam", "mean", "rstd"):
            assert torch.equal(out[k], want[k]), (k, stages, park)
    assert nt.wait_timeouts() == 0


@pytest.mark.parametrize("N,C,sp,G,dt,ctas", [
    (1, 1024, (37, 5), 128, "float16", 3),    # the most groups, a vector each: four threads to a group
    (2, 512, (29, 7), 128, "float32", 4),     # the same with four lanes
    (1, 128, (61, 3), 128, "bfloat16", 2),    # one channel per group, 32 row lanes
    (1, 24, (331, 5), 3, "bfloat16", 2),      # three groups, 170 row lanes, two idle threads
    (1, 240, (47, 9), 30, "float16", 2),      # 17 row lanes of 30 threads: half a warp without work
    (2, 264, (31, 11), 3, "float16", 3),      # eleven vectors per group
    (1, 2048, (19, 3), 1, "float32", 2),      # one row lane of 512 threads
    (1, 40, (3, 1), 8, "float16", 2),         # fewer rows than row lanes
], ids=lambda v: str(v).replace(" ", ""))
def test_reductions_over_the_cta(N, C, sp, G, dt, ctas, monkeypatch):
    """csrc/gn_reduce.cuh: group moments, channel sums and group sums at the edges of its layout, against the fp64 oracle."""
    from channels_last_groupnorm_b200 import _native as nt

    monkeypatch.setenv("GNB200_FORCE_PATH", "resident")
    monkeypatch.setenv("GNB200_RESIDENT_CTAS", str(ctas))
    assert " resident=1 " in nt.describe_plan(N, sp[0] * sp[1], C, G, DT[dt], 0)
    x, ga, be, dy = O.make_inputs(N, C, sp, DT[dt], seed=31, x_dist="uniform3")
    out = run_cabi(nt, x, ga, be, dy, G, 1e-5, "silu")
    want = O.oracle_c(x, ga, be, dy, G, 1e-5, "silu", threads=4)
    check_against(out, want, DT[dt])
    # fp32 sums over at most a few thousand values of one group or channel
    assert O.rel_err(out["mean"], want["mean"]) < 1e-5
    assert O.rel_err(out["rstd"] / want["rstd"].cuda().float(), torch.ones_like(want["rstd"])) < 1e-5
    assert O.rel_err(out["dparam"][0], want["dgamma"]) <= O.TOLERANCE[DT[dt]] and O.rel_err(out["dparam"][1], want["dbeta"]) <= O.TOLERANCE[DT[dt]]


@pytest.mark.parametrize("what", [3, 4, 5], ids=["no arrival", "no first copy", "no copy of the second pass"])
@pytest.mark.parametrize("dt,act", [("float16", "silu"), ("float32", "relu")])
def test_waits_that_run_out_with_tiles_in_tensor_memory(what, dt, act, monkeypatch):
    """One CTA withholds what others, or its own threads, wait for (decided on the host, wait limit one millisecond) while tiles are
    in tensor memory.  The call returns, what depends on it is NaN, the parked rows of a lost second pass are not, and the
    tensor memory is given back: the next calls get it and have the bits of the first."""
    from channels_last_groupnorm_b200 import _native as nt

    from .test_parity_gpu import _flat

    N, C, sp, G, code, ctas, cta, park = 2, 64, (32, 240), 8, O.ACT_CODES[act], 3, 1, 3
    for name, value in (("FORCE_PATH", "resident"), ("RESIDENT_CTAS", ctas), ("RESIDENT_STAGES", 2), ("RESIDENT_PARK", park)):
        monkeypatch.setenv("GNB200_" + name, str(value))
    x, ga, be, dy = O.make_inputs(N, C, sp, DT[dt], seed=61)
    xd, dyd, gd, bd = _flat(x.cuda()), _flat(dy.cuda()), ga.cuda(), be.cuda()
    good = nt.fwd_raw(xd, gd, bd, G, 1e-5, code)
    calls = (lambda: nt.fwd_raw(xd, gd, bd, G, 1e-5, code), lambda: nt.bwd_raw(dyd, xd, gd, bd, good[1], good[2], G, code))
    for direction in (0, 1):
        want = calls[direction]()
        nt.check(nt.lib.gnb200_debug_next_resident(what, cta))
        try:
            got = calls[direction]()
            torch.cuda.synchronize()  # the call returns and the GPU still answers
            assert nt.wait_timeouts() > 0
        finally:
            nt.clear_wait_timeouts()
        if what != 5:
            assert all(torch.isnan(t.float()).all() for t in got)
        else:  # two tiles were in the stages and `park` in tensor memory: those before them are missing
            plan = dict(kv.split("=") for kv in nt.describe_plan(N, sp[0] * sp[1], C, G, DT[dt], direction).split()[2:])
            rows, tile = int(plan["rows"]), int(plan["tile"].split("x")[1])
            tiles = -(-rows // tile)
            assert tiles > 2 + park
            missing = torch.zeros(sp[0] * sp[1], dtype=torch.bool, device="cuda")
            missing[cta * rows:cta * rows + (tiles - 2 - park) * tile] = True
            assert torch.isnan(got[0][0, missing].float()).all()
            assert torch.equal(got[0][0, ~missing], want[0][0, ~missing]) and torch.equal(got[0][1], want[0][1])
        for _ in range(3):
            assert all(torch.equal(a, b) for a, b in zip(calls[direction](), want))
    assert nt.wait_timeouts() == 0
