"""The plain walk's term list holds 64 entries: a walk that meets overflow
buckets (several particles in one cell of the deepest level) in any round
stays within it and evaluates every particle once for every target."""
import numpy as np
import pytest

import plain_list_model as pm


def clustered(seed, n=2001, clusters=10, size=40):
    rng = np.random.default_rng(seed)
    x = 1.0 + rng.uniform(-0.5, 0.5, size=(n, 3))
    for c in range(clusters):  # within a fraction of 2 / 2^21, one deepest cell (rarely two)
        a = 10 + (n // clusters - 5) * c
        x[a:a + size] = x[a] + rng.uniform(0.0, 1e-9, size=(size, 3))
    return x


def cases(seed):
    x = clustered(seed)
    t = pm.tree(x, 2.0)
    rng = np.random.default_rng(100 + seed)
    for g, theta in ((2, 1e-7), (4, 1e-7), (8, 1e-7), (8, 0.3)):
        a = int(rng.integers(0, len(x) - g))
        yield x, t, list(range(a, a + g)), theta


@pytest.mark.parametrize("seed", range(6))
def test_list_stays_within_its_entries(seed):
    for x, t, targets, theta in cases(seed):
        high, done = pm.walk(t, x, targets, theta)
        assert high < pm.LIST, high
        if theta > 0.01:
            continue
        # every cell opens: each target's terms are all other particles, once each
        for k, me in enumerate(targets):
            terms = sorted(e[1] for e, m in done if (m >> k) & 1)
            assert terms == [i for i in range(len(x)) if i != me]


def test_a_round_with_a_bucket_needs_the_list_flushed_first():
    """The premise: in the same walks a bucket appended to a list that is not
    evaluated first would go past the list."""
    high = max(pm.walk(t, x, targets, theta, flush_before_buckets=False)[0]
               for seed in range(6) for x, t, targets, theta in cases(seed))
    assert high >= pm.LIST, high
