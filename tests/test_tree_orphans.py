"""A tree over keys that are out of order (a radix sort whose look-back gave up
sets POT_E_ITER and goes on) can hold cells that no parent claims, whose entry
of T.parent is whatever the memory held.  Restates the claims of k_finish_nodes
and the uses of the entry in the moments kernels (pot_tree.cu): no index taken
from it leaves its array."""
import os
import re

import numpy as np
import pytest

import tree_model as tm

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pot_b200", "csrc", "pot_tree.cu")


def parents(keys, garbage, L=1):
    """T.parent after the topology kernels (plain form: the parent cell; fast
    form: the cell's record, as many in number), garbage where nobody wrote."""
    n = len(keys)
    lvl = np.minimum(tm.lcp_levels(keys[:n - L], keys[L:]), tm.MAX_LEVELS - 1)
    prev = np.concatenate([[-1], lvl[:-1]])
    cnt = np.maximum(lvl - prev, 0)
    base = np.concatenate([[0], np.cumsum(cnt)[:-1]])
    M = int(cnt.sum())
    first = np.repeat(np.arange(n - L), cnt)
    level = np.concatenate([np.arange(p + 1, l + 1) for p, l in zip(prev, lvl)])
    out = np.array(garbage[:M])
    claimed = set()
    for k in range(M):
        f, l = int(first[k]), int(level[k])
        shift = 63 - 3 * l
        e = tm.cell_end(keys, f, n, shift, int(keys[f]) >> shift)
        s = [f] + tm.child_starts(keys, f, e, shift - 3) + [e]
        for d in range(8):
            c = int(s[d + 1]) - int(s[d])
            if 0 <= c <= L or l + 1 >= tm.MAX_LEVELS:
                continue
            sc = int(s[d])
            lo = 0 if sc == 0 or sc > len(lvl) else int(lvl[sc - 1]) + 1
            if sc + L >= n:
                continue
            kc = int(base[sc]) + l + 1 - lo
            if kc < 0 or kc >= M or kc <= k:
                continue
            out[kc] = k
            claimed.add(kc)
    out[0] = -1
    return out, len(claimed), M


def test_unclaimed_cells_are_not_followed():
    rng = np.random.default_rng(1)
    x, y, z = rng.uniform(0.0, 1.0, size=(3, 400))
    keys = np.sort(tm.morton_keys(x, y, z, 1.0))
    _, claimed, M = parents(keys, np.zeros(4000, np.int64))
    assert claimed == M - 1  # in order: every cell but the root
    orphans = wild = 0
    for seed in range(4):
        shuffled = np.random.default_rng(seed).permutation(keys)
        garbage = rng.integers(-2 ** 31, 2 ** 31, size=4000)
        par, claimed, M = parents(shuffled, garbage)
        cap = 4 * len(keys) + 4096
        assert M <= cap
        orphans += M - 1 - claimed
        spare = 1 + cap + len(keys)
        for k in range(1, M):
            # k_moments: nint[p], cells p < k only
            p = int(par[k])
            orphan = p < 0 or p >= k
            assert orphan or p < M
            # moments_prefix_body: nrec[o], records up to the spare one
            o = min(int(par[k]) & 0xFFFFFFFF, spare)
            assert 0 <= o <= spare
            wild += int(par[k]) & 0xFFFFFFFF > spare
    assert orphans > 0 and wild > 0  # without the checks these were followed


def test_a_sort_that_gave_up_leaves_indices_of_particles():
    """A tile whose look-back stops early counts too few of the earlier tiles'
    keys: it writes over theirs, never past its digit, and leaves other slots
    with what they held.  That is an index too: the keys kernel writes one order
    every step and a context starts with the other cleared."""
    rng = np.random.default_rng(2)
    n, tile = 20000, 2048
    vals = [np.arange(n), np.zeros(n, np.int64)]
    unwritten = 0
    for step in range(3):
        vals[0] = np.arange(n)
        for p in range(4):
            src, dst = vals[p & 1], vals[(p + 1) & 1]
            digit = rng.integers(0, 256, n)
            start = np.concatenate([[0], np.cumsum(np.bincount(digit, minlength=256))])
            written = np.zeros(n, bool)
            for t0 in range(0, n, tile):
                seen = int(rng.integers(0, t0 // tile + 1)) * tile  # the tiles the look-back reached
                before = np.bincount(digit[t0 - seen:t0], minlength=256)
                count = np.zeros(256, int)
                for i, d in enumerate(digit[t0:t0 + tile]):
                    o = start[d] + before[d] + count[d]
                    assert o < start[d + 1]
                    dst[o] = src[t0 + i]
                    written[o] = True
                    count[d] += 1
            unwritten += int((~written).sum())
            assert dst.min() >= 0 and dst.max() < n
    assert unwritten > 0  # the premise
    api = open(os.path.join(os.path.dirname(SRC), "pot_api.cu")).read()
    assert "cudaMemsetAsync(c->vals[1], 0, sizeof(uint32_t) * n, c->stream)" in api


@pytest.mark.parametrize("use,check", [(r"T\.nint\[p\]", r"\(uint32_t\)p >= k"), (r"T\.nrec\[o\]", r"o = [^;]*min\([^;]*, spare\);")])
def test_checks_stand_ahead_of_the_uses(use, check):
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    uses = [m.start() for m in re.finditer(use, text)]
    assert uses
    for u in uses:
        assert re.search(check, text[max(0, u - 1500):u]), use
