"""The fast walk's node records at their edges: leaves of one particle and of
buckets far above the leaf size (cells of the deepest level), for one and two
targets per lane, with every cell opened so that the walk is a direct sum."""
from __future__ import annotations

import numpy as np
import pytest

from pot_b200.gpu import PARTICLE_DTYPE, Run
from tests.common import SMALL, run_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf,group", [(1, 32), (1, 64), (4, 32), (16, 32), (16, 64)])
@pytest.mark.parametrize("N", [34, 603])
def test_opened_fast_tree_is_a_direct_sum(N, leaf, group):
    R = SMALL["r"] * SMALL["mpp"]
    d = dict(SMALL, theta=1e-6, soft=0.05 * R)
    rng = np.random.default_rng(N)
    x = R + rng.uniform(-0.5 * R, 0.5 * R, size=(N, 3))
    if N > 100:  # three clusters of 70, each inside one cell of the deepest level
        for c in range(3):
            x[10 + 150 * c:80 + 150 * c] = x[10 + 150 * c] + rng.uniform(0.0, 1e-9 * R, size=(70, 3))
    x[0] = R
    p = np.zeros(N, PARTICLE_DTYPE)
    for k, a in enumerate("xyz"):
        p[a] = x[:, k]
    p["species"][1:] = np.where(np.arange(N - 1) < (N - 1) // 2, 1, 2)
    q = np.where(p["species"] == 1, 1.0, -1.0)
    q[0] = -7.0
    dx = x[:, None, :] - x[None, :, :]
    r2 = (dx ** 2).sum(-1) + d["soft"] ** 2
    term = 1.6021766e-19 / (4 * 3.14159265358979 * 8.85419e-12) * q[None, :, None] * dx / r2[:, :, None] ** 1.5
    ref, scale = term.sum(1), np.linalg.norm(np.abs(term).sum(1), axis=1)
    with Run(run_config(d, N=N), form="fast", leaf_size=leaf, group_size=group) as r:
        r.upload(p, dict(q=-7, pos=tuple(x[0])))
        r.build_tree()
        E = r.field_at(np.arange(N, dtype=np.uint32), x)
    # N terms of FP32 rounding (6e-8) each, against the sum of their magnitudes
    assert (np.linalg.norm(E - ref, axis=1) <= 5e-5 * scale).all()
