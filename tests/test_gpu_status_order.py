"""Which status a state with several faults ends with, on a step replayed as a
graph, whose branches run side by side: the one the launches' order gives."""
from __future__ import annotations

import numpy as np
import pytest

from pot_b200.gpu import PARTICLE_DTYPE, PotError, Run
from tests.common import SMALL, run_config

pytestmark = pytest.mark.gpu

E_COINCIDENT, E_WALK, E_CAPACITY = -5, -6, -9


def _state(N, R, seed):
    rng = np.random.default_rng(seed)
    x = R + rng.uniform(-0.5 * R, 0.5 * R, size=(N, 3))
    x[0] = R
    p = np.zeros(N, PARTICLE_DTYPE)
    for k, a in enumerate("xyz"):
        p[a] = x[:, k]
    p["species"][1:] = np.where(np.arange(N - 1) < (N - 1) // 2, 1, 2)
    return p


@pytest.mark.parametrize("form,leaf", [("plain", 1), ("fast", 1)])
def test_coincident_particles_are_reported_first(form, leaf):
    """6,000 pairs share deepest cells (more than the overflow buckets hold:
    the tree is too large) and the last two particles share a position."""
    N = 400001
    d = dict(SMALL, N=N)
    R = d["r"] * d["mpp"]
    good = _state(N, R, 1)
    bad = _state(N, R, 2)
    for a in "xyz":
        bad[a][1:6001] = R - 0.5 * (R - bad[a][1:6001]) - 0.25 * R  # near the first corner
        bad[a][6001:12001] = bad[a][1:6001] * (1.0 + 2.0 ** -40)
    full = bad.copy()
    for a in "xyz":
        bad[a][N - 2] = bad[a][N - 1] = 1.55 * R
    with Run(run_config(d), form=form, leaf_size=leaf) as r:
        r.upload(good)
        r.step(6)  # both parities captured
        for p, want in ((full, E_CAPACITY), (bad, E_COINCIDENT), (bad, E_COINCIDENT), (bad, E_COINCIDENT)):
            r.upload(p)
            with pytest.raises(PotError) as e:
                r.step(1)
            assert e.value.status == want
        r.upload(good)
        r.step(2)


@pytest.mark.parametrize("leaf", [1, 8, 64])
@pytest.mark.parametrize("where", [0.48, 1.56], ids=["first", "last"])
def test_coincident_neighbours_at_the_ends(leaf, where):
    """The first and the last slots' neighbours, which the pairs (i, i + leaf)
    do not all cover."""
    N = 5000
    d = dict(SMALL, N=N)
    R = d["r"] * d["mpp"]
    p = _state(N, R, 3)
    for a in "xyz":
        p[a][N - 2] = p[a][N - 1] = where * R
    with Run(run_config(d), form="fast", leaf_size=leaf) as r:
        r.upload(p)
        with pytest.raises(PotError) as e:
            r.build_tree()
        assert e.value.status == E_COINCIDENT


@pytest.mark.parametrize("form,N", [("plain", 20001), ("fast", 20001), ("fast", 2000001)])
def test_a_failed_edge_potential_stops_the_push(form, N):
    """An edge potential that is no number (the grain's position given as NaN) on
    the 20th step: the step ends with the walk's status and no particle moves."""
    d = dict(SMALL, N=N)
    p = _state(N, d["r"] * d["mpp"], 4)
    c = (p["x"][0], p["y"][0], p["z"][0])
    rng = np.random.default_rng(5)
    for a in ("vx", "vy", "vz"):
        p[a][1:] = rng.normal(0.0, 4e5, N - 1)
    with Run(run_config(d), form=form) as r:
        r.upload(p, dict(q=-7, pos=c, t_steps=2))
        r.step(6)  # both parities captured
        for _ in range(3):
            r.upload(p, dict(q=-7, pos=c, t_steps=18))
            r.step(1)
            out, _ = r.download()
            r.upload(out, dict(q=-7, pos=(np.nan, c[1], c[2]), t_steps=19))
            with pytest.raises(PotError) as e:
                r.step(1)
            assert e.value.status == E_WALK
            assert e.value.stats["n_pushed"] == 0
