"""Which status a state with several faults ends with, on a step replayed as a
graph, whose branches run side by side: the one the launches' order gives."""
from __future__ import annotations

import numpy as np
import pytest

from pot_b200.gpu import PARTICLE_DTYPE, PotError, Run
from tests.common import SMALL, run_config

pytestmark = pytest.mark.gpu

E_COINCIDENT, E_CAPACITY = -5, -9


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
