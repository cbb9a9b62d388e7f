"""Plans come from a per-thread table unless an override is set: the table must not mix problems up, and an override
set later must be seen."""
import os
import random
import re
import threading
import time

import pytest
import torch

from channels_last_groupnorm_b200 import _native as nt

DTYPES = [torch.float32, torch.float16, torch.bfloat16]


def _problems(seed, count):
    rng = random.Random(seed)
    for _ in range(count):
        g = rng.choice([1, 3, 8, 32])
        yield (rng.choice([1, 2, 16]), rng.choice([1, 49, 1000, 4096, 70000]), g * rng.choice([1, 5, 8, 10, 40]), g,
               rng.choice(DTYPES), rng.choice([0, 1]))


def test_remembered_plans_equal_fresh_ones(monkeypatch):
    problems = list(_problems(3, 300))  # several times the size of the table: entries are replaced
    first = [nt.describe_plan(*p) for p in problems]
    again = [nt.describe_plan(*p) for p in problems]
    monkeypatch.setenv("GNB200_CHAIN", "1")  # any override: every plan is made anew (this one changes nothing)
    fresh = [nt.describe_plan(*p) for p in problems]
    assert first == again == fresh


def test_an_override_is_seen_after_a_plan_was_remembered(monkeypatch):
    before = nt.describe_plan(2, 1024, 128, 32, torch.float32, 0)
    monkeypatch.setenv("GNB200_FORCE_PATH", "twopass")
    assert " twopass " in nt.describe_plan(2, 1024, 128, 32, torch.float32, 0)
    monkeypatch.delenv("GNB200_FORCE_PATH")
    assert nt.describe_plan(2, 1024, 128, 32, torch.float32, 0) == before and " fused " in before


def test_threads_make_the_same_plans():
    problems = list(_problems(5, 100))
    want = [nt.describe_plan(*p) for p in problems]
    got = {}
    threads = [threading.Thread(target=lambda i=i: got.__setitem__(i, [nt.describe_plan(*p) for p in problems])) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(got[i] == want for i in range(4))


def _query_time():
    best = 1e9
    for _ in range(20):
        t0 = time.perf_counter()
        for _ in range(50):
            nt.lib.gnb200_bwd_workspace_bytes(1, 65536, 512, 32, 1)
        best = min(best, (time.perf_counter() - t0) / 50)
    return best


@pytest.mark.parametrize("name", ["GNB200_WAIT_CLOCKS", "GNB200_PEER_LANES"])
def test_variables_that_are_no_override_leave_the_table_on(name, monkeypatch):
    """A query makes two plans: some 20 us searched anew, under 2 us from the table."""
    plain = _query_time()
    monkeypatch.setenv("GNB200_CHAIN", "1")
    searched = _query_time()
    monkeypatch.delenv("GNB200_CHAIN")
    monkeypatch.setenv(name, "32")
    with_it = _query_time()
    assert searched > 3 * plain and with_it < 0.5 * (plain + searched), (plain, searched, with_it)


def test_every_name_the_planner_reads_counts_as_an_override(repo_root):
    text = open(os.path.join(repo_root, "channels_last_groupnorm_b200", "csrc", "gn_plan.cu")).read()
    read = set(re.findall(r'env_(?:int|text)\("GNB200_(\w+)"', text))
    known = re.findall(r'"(\w+=?)"', re.search(r"kOverrides\[\] = \{(.*?)\};", text, re.S).group(1))
    assert len(read) > 10
    for name in read:
        assert any((name + "=").startswith(k) for k in known), name
