"""CPU tests of the rule that takes a call to the resident plan (csrc/gn_resident.cu) without any override."""
import random

import pytest
import torch

from channels_last_groupnorm_b200 import _native as nt

F16, BF16, F32 = torch.float16, torch.bfloat16, torch.float32


def _fields(text):
    return dict(kv.split("=") for kv in text.split()[2:])


# per direction, both sides of every line of the rule; shapes beyond a cluster, so that only the rule decides
MB48 = 48 * 1024 * 1024
RULE = [
    # direction, (N, R, C, G, dtype), resident?
    (0, (1, MB48 // 512, 256, 8, F16), True),         # one 16-bit sample of 48 MB and eight groups ...
    (0, (1, MB48 // 512 - 1, 256, 8, F16), False),    # ... and a row less
    (0, (1, MB48 // 512, 256, 8, BF16), True),
    (0, (2, MB48 // 512, 256, 8, F16), False),        # two samples
    (0, (1, MB48 // 512, 256, 8, F32), False),        # fp32
    (0, (1, MB48 // 512, 256, 4, F16), False),        # four groups
    (0, (1, 1 << 18, 2048, 128, F16), True),          # 128 groups at most: every CTA merges all partial sums
    (0, (1, 1 << 18, 4096, 256, F16), False),
    (0, (1, 1 << 22, 20, 10, F16), False),            # rows that are not whole 16-byte vectors
    (1, (1, 1 << 18, 256, 32, F16), True),
    (1, (3, 1 << 17, 256, 32, BF16), True),
    (1, (1, 1 << 18, 256, 32, F32), False),           # fp32 only with 128 channels per group
    (1, (1, 1 << 17, 512, 4, F32), True),
    (1, (1, 1 << 17, 508, 4, F32), False),
    (1, (1, 1 << 18, 256, 256, F16), False),
    (1, (1, 1 << 18, 4096, 32, F16), False),          # scratch above 4 MiB and 33 KB more than the wave plan's
    (1, (1, 1 << 18, 4104, 27, F16), False),          # 513
    (1, (21, 1 << 17, 64, 1, F16), True),             # 21 x 7 = 147 of 148 CTAs
    (1, (30, 1 << 17, 64, 1, F16), False),            # 30 x 4 = 120, below 85 %
    (1, (149, 1 << 15, 64, 1, F16), False),           # more samples than SMs
    (1, (1, 149, 4096, 1, F16), True),                # two rows per CTA: 75 CTAs, and still the better plan
    (1, (1, 4096, 4096, 1, F16), True),               # 28 rows per CTA: 147; 512 vectors per row, the most
]


@pytest.mark.parametrize("direction,shape,want", RULE, ids=lambda v: "-".join(map(str, v)).replace("torch.", "") if isinstance(v, tuple) else str(v))
def test_which_calls_take_the_resident_plan(direction, shape, want):
    text = nt.describe_plan(*shape, direction)
    assert (_fields(text).get("resident") == "1") is want, text
    assert " fused " not in text


def test_scratch_of_the_resident_plan_stays_within_the_callers_limits():
    """Never less than the plan it stands in for asks for, and beyond 4 MiB (the scratch that every backward may rely on)
    never more; the query covers it, and the grid fits the SMs."""
    rng = random.Random(11)
    seen = 0
    for _ in range(3000):
        G = rng.choice([1, 2, 8, 32, 64])
        C = G * rng.choice([1, 2, 8, 10, 16, 40, 64, 512, 4096])
        N, R, dtype, direction = rng.choice([1, 2, 3, 20]), rng.choice([149, 1000, 5000, 70000, 1 << 18]), rng.choice([F16, BF16, F32]), rng.choice([0, 1])
        if C > 8192 or N * R * C > 1 << 31:
            continue
        text = nt.describe_plan(N, R, C, G, dtype, direction)
        f = _fields(text)
        if f.get("resident") != "1":
            continue
        seen += 1
        ws = int(f["ws"])
        query = nt.lib.gnb200_fwd_workspace_bytes if direction == 0 else nt.lib.gnb200_bwd_workspace_bytes
        assert ws <= query(N, R, C, G, nt.DTYPE_CODES[dtype]) and int(f["grid"]) <= 148
        own = int(f["grid"]) * (G * 8 + (C * 8 if direction else 0)) + 4
        assert ws >= own
        with pytest.MonkeyPatch.context() as mp:
            mp.setenv("GNB200_FORCE_PATH", "wave" if f["fallback"] == "wave" else "twopass")
            other = int(_fields(nt.describe_plan(N, R, C, G, dtype, direction))["ws"])
        assert ws >= other and (ws == other or ws <= 4 << 20), text
    assert seen > 200
