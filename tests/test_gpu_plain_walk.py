"""The plain form's shared walk at the edges of its shapes: targets per warp
(2, 4 or 8 by the number of targets), partial groups, overflow buckets and a
stack kept within its capacity."""
from __future__ import annotations

import numpy as np
import pytest

from oracle.oracle import Oracle
from pot_b200.gpu import PARTICLE_DTYPE, Run
from tests.common import SMALL, ld, oracle_snapshot, params, run_config

pytestmark = pytest.mark.gpu


def _upload(d, p, q, **over):
    r = Run(run_config(d, N=len(p), **over), form="plain")
    r.upload(p, dict(q=q, pos=(p["x"][0], p["y"][0], p["z"][0])))
    r.build_tree()
    return r


@pytest.mark.parametrize("dipoles", [False, True], ids=["monopoles", "dipoles"])
@pytest.mark.parametrize("nq", [1, 3, 8191, 8193, 32769])
def test_field_for_every_group_size(nq, dipoles):
    if dipoles and nq > 3:
        pytest.skip("one group size with dipoles")
    o = oracle_snapshot(SMALL, seed=4, dipoles=dipoles)
    o.set_grain(q=-250)
    o.build_tree()
    p = o.particles()
    rng = np.random.default_rng(nq)
    # neighbours, strangers, the grain and points that belong to no particle
    idx = np.sort(rng.integers(0, SMALL["N"], nq)).astype(np.uint32)
    idx[0] = 0
    xyz = np.stack([p[a][idx] for a in "xyz"], 1)
    hi, lo = o.field_many(idx, xyz)
    ref = ld(hi, lo).astype(np.float64)
    with _upload(SMALL, p, -250, dipoles=dipoles) as r:
        E = r.field_at(idx, xyz)
    # 1,000 terms of FP64 rounding each against a sum whose parts cancel
    err = np.abs(E - ref).max(1) / np.linalg.norm(ref, axis=1)
    assert err.max() < 1e-12, err.max()


@pytest.mark.parametrize("N", [2, 3, 35, 601])
def test_opened_tree_with_overflow_buckets(N):
    """An opening angle at which nearly every cell opens (the stack's cap) and
    clusters inside one cell of the deepest level (buckets of up to 40)."""
    d = dict(SMALL, theta=1e-4)
    R = d["r"] * d["mpp"]
    rng = np.random.default_rng(N)
    x = R + rng.uniform(-0.5 * R, 0.5 * R, size=(N, 3))
    if N > 100:
        for c in range(3):  # 40 particles within a fraction of 2 R / 2^21
            x[10 + 100 * c:50 + 100 * c] = x[10 + 100 * c] + rng.uniform(0.0, 1e-9 * R, size=(40, 3))
    x[0] = R
    p = np.zeros(N, PARTICLE_DTYPE)
    for k, a in enumerate("xyz"):
        p[a] = x[:, k]
    p["species"][1:] = np.where(np.arange(N - 1) < (N - 1) // 2, 1, 2)
    o = Oracle(params(d, N=N), mode="gpu", sceptic=True, seed=1)
    o.set_particles(p)
    o.set_grain(q=-7)
    o.build_tree()  # splits the clusters' cells further: the same terms, all of them pairs
    idx = np.arange(N, dtype=np.uint32)
    hi, lo = o.field_many(idx, x)
    ref = ld(hi, lo).astype(np.float64)
    q = np.where(p["species"] == 1, 1.0, -1.0)
    q[0] = -7.0
    dx = x[:, None, :] - x[None, :, :]
    r2 = (dx ** 2).sum(-1) + d["soft"] ** 2
    np.fill_diagonal(r2, np.inf)
    k = 1.6021766e-19 / (4 * 3.14159265358979 * 8.85419e-12)
    scale = np.linalg.norm(np.abs(k * q[None, :, None] * dx / r2[:, :, None] ** 1.5).sum(1), axis=1)
    with _upload(d, p, -7) as r:
        E = r.field_at(idx, x)
    # every term within a few roundings, N of them: relative to the sum of magnitudes
    assert np.abs(E - ref).max(1).max() < 1e-12 * scale.max()
    assert (np.linalg.norm(E - ref, axis=1) <= 1e-13 * scale).all()
