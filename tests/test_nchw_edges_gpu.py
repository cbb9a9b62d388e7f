"""Channels-first kernels at the edges of their split: the output passes walk chunks and pieces backwards, and the
channel sums are gathered a lane per piece (more than 32 pieces for long rows)."""
import pytest
import torch

from oracle import gn_oracle as O

from .test_nchw_f64_gpu import DT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [
    (1, 4, (128, 264), 2, "float16", "silu"),      # rows of 4224 vectors: more than 32 pieces per row
    (1, 3, (61, 67), 3, "float32", "gelu"),        # single elements, ragged last piece
    (2, 6, (8, 12), 1, "bfloat16", "relu"),        # rows of 12 vectors: one piece, idle lanes
    (1, 33, (32, 40), 1, "float16", "gelu_tanh"),  # one group of 33 channels: warps take unequal shares
    (1, 2, (1, 8), 1, "float16", "identity"),      # one vector per row
    (1, 8, (200, 331), 1, "float32", "silu"),      # many chunks per slab, remainder at both ends
    (1, 8, (64, 98), 1, "float16", "silu"),        # 6272 vectors: three chunks of two whole batches and a rest of 128
    (1, 6, (61, 67), 2, "bfloat16", "gelu"),       # 12261 single elements: chunks of 4096, four batches
    (1, 2048, (24, 25), 32, "float32", "silu"),    # 2048 rows of 150 vectors: pieces of 256 at least, so one of 160
    (2, 8, (100, 92), 2, "float16", "relu"),       # rows of 1150 vectors: nine equal pieces, the last one shorter
], ids=lambda c: "%dx%dx%s-g%d-%s-%s" % (c[0], c[1], "x".join(map(str, c[2])), *c[3:]))
def test_channels_first_edges_against_oracle(case):
    from channels_last_groupnorm_b200 import _native as nt

    N, C, sp, G, dt, act = case
    x, ga, be, dy = O.make_inputs(N, C, sp, DT[dt], seed=31, x_dist="uniform3")
    flat = lambda t: t.contiguous().reshape(N, C, -1).cuda()
    code = O.ACT_CODES[act]
    y, mean, rstd = nt.fwd_nchw_raw(flat(x), ga.cuda(), be.cuda(), G, 1e-5, code)
    dx, dparam, dgamma, dbeta = nt.bwd_nchw_raw(flat(dy), flat(x), ga.cuda(), be.cuda(), mean, rstd, G, code)
    want = O.oracle_c(x, ga, be, dy, G, 1e-5, act, threads=4)
    tol = O.TOLERANCE[DT[dt]]
    assert O.rel_err(y.reshape(N, C, *sp), want["y"]) <= tol and O.rel_err(dx.reshape(N, C, *sp), want["dx"]) <= tol
    assert O.rel_err(dparam[0], want["dgamma"]) <= tol and O.rel_err(dparam[1], want["dbeta"]) <= tol
    assert O.rel_err(mean, want["mean"]) < 1e-5
