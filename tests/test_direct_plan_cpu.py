"""The one-launch kernel's work list: every row sees every one of its tokens exactly once, whatever the tree, and tokens
appended after the list was made are seen, too.  Runs without a GPU."""
import random

import numpy as np
import pytest

from chunk_attn import cabi
from test_plan_cpu import build_tree, plan_of, shared_spec

STEP, WARPS, TO_THE_END = 16, 4, 1 << 20


def walk(plan, cluster, n_seqs, chunk_size, delta):
    """What the kernel's warps do: {row: [(chunk, token), ...]}."""
    entries = plan.array(cabi.PLAN_DIRECT_ENTRIES).reshape(-1, 4)
    blocks = plan.array(cabi.PLAN_DIRECT_BLOCKS).reshape(-1, 2)
    ranges = plan.array(cabi.PLAN_DIRECT_RANGES).reshape(len(blocks), cluster * WARPS, 4)
    seen = {r: [] for r in range(n_seqs)}
    for (row0, rows), warps in zip(blocks, ranges):
        assert 1 <= rows <= 8
        for e0, s0, e1, s1 in warps:
            for e in range(e0, e1 + 1):
                chunk, n, mask, tail = entries[e]
                n = min(chunk_size, n + (delta if tail else 0))
                assert 0 < mask < 1 << rows
                for t in range(s0 * STEP if e == e0 else 0, min(n, s1 * STEP) if e == e1 else n):
                    for r in range(rows):
                        if mask >> r & 1:
                            seen[row0 + r].append((int(chunk), t))
    assert sorted(r for b, n in blocks for r in range(b, b + n)) == list(range(n_seqs))
    return seen


def expected(ora, delta):
    want = {}
    for r in range(len(ora.tails)):
        path = [(c, b, e) for c, b, e in ora.get_chunks() if b <= r < e]
        want[r] = sorted((c.id, t) for i, (c, _, _) in enumerate(path)
                         for t in range(min(ora.chunk_size, c.n_tokens + delta) if i == len(path) - 1 else c.n_tokens))
    return want


def random_spec(rng, n):
    """Prompts that share prefixes of prefixes."""
    spec = []
    for i in range(n):
        base = rng.choice(spec) if spec and rng.random() < 0.7 else []
        spec.append(list(base[:rng.randint(0, len(base))]) + [1000 * (i + 1) + j for j in range(rng.choice([1, 2, 15, 16, 17, 40, 64, 100, 200]))])
    return spec


@pytest.mark.parametrize("seed", range(12))
def test_every_token_once(seed):
    rng = random.Random(seed)
    chunk = rng.choice([16, 24, 32, 40, 64])
    spec = random_spec(rng, rng.choice([1, 2, 3, 7, 8, 9, 17, 40]))
    heads = rng.choice([1, 4, 32])
    ora = build_tree(spec, seed=seed, chunk_size=chunk)
    plan, _ = plan_of(ora, heads)
    cluster = plan.direct(2, rng.choice([32, 64, 128]), against_items=bool(seed & 1))
    assert cluster in (1, 2, 4, 8)
    for delta in (0, 1, 3, STEP, chunk):
        seen = walk(plan, cluster, len(ora.tails), chunk, delta)
        want = expected(ora, delta)
        for r in want:
            assert sorted(seen[r]) == want[r], (r, delta)


def test_empty_tails_take_their_first_token():
    ora = build_tree([list(range(64)) + [1000 + i] for i in range(3)] + [list(range(64))])
    ora.reserve()
    plan, _ = plan_of(ora, 4)
    cluster = plan.direct(2, 128)
    for delta in (0, 1):
        assert {r: sorted(s) for r, s in walk(plan, cluster, len(ora.tails), 64, delta).items()} == expected(ora, delta)


def test_which_way():
    # a few short rows go the one-launch way, large steps and many short tails do not, off is off
    small, _ = plan_of(build_tree(shared_spec(4, 128, 100)), 8)
    assert small.direct(1, 128) > 0 and small.direct(0, 128) == 0
    assert small.array(cabi.PLAN_DIRECT_ENTRIES).size == 0
    large, _ = plan_of(build_tree(shared_spec(64, 0, 2200)), 32)
    assert large.direct(1, 128) == 0 and large.direct(2, 128) > 0
    tails, _ = plan_of(build_tree(shared_spec(300, 128, 4)), 8)
    assert tails.stats()["n_items_short"] > 0 and tails.direct(1, 128) == 0
    # where the any-geometry kernel is the alternative, the smallest steps are its own
    least, _ = plan_of(build_tree(shared_spec(7, 128, 21), chunk_size=16), 1)
    assert least.direct(1, 64, against_items=False) == 0 and least.direct(2, 64, against_items=False) > 0
    few, _ = plan_of(build_tree(shared_spec(7, 0, 10)), 8)
    assert few.direct(1, 64, against_items=False) == 0
    over, _ = plan_of(build_tree(shared_spec(54, 1024, 49), chunk_size=16), 16)
    assert over.direct(1, 64, against_items=False) > 0
    with pytest.raises(cabi.CAError):
        small.direct(1, 256)
    with pytest.raises(cabi.CAError):
        small.direct(3, 128)
