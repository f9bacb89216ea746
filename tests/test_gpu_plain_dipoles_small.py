"""The plain walk with dipoles where its term list is never full: trees of a
few particles whose cells all open, queried right after a larger run's
potential query has left its stack of leaf codes (as doubles, NaN) in the shared
memory the lists lie in."""
from __future__ import annotations

import numpy as np
import pytest

from pot_b200.gpu import PARTICLE_DTYPE, Run
from tests.common import SMALL, oracle_snapshot, run_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [2, 3, 35, 70])
def test_opened_tree(N):
    o = oracle_snapshot(SMALL, seed=2)
    big = o.particles()
    d = dict(SMALL, N=N, theta=1e-9)
    R = d["r"] * d["mpp"]
    rng = np.random.default_rng(N)
    x = R + rng.uniform(-0.5 * R, 0.5 * R, size=(N, 3))
    p = np.zeros(N, PARTICLE_DTYPE)
    for k, a in enumerate("xyz"):
        p[a] = x[:, k]
    p["species"][1:] = np.where(np.arange(N - 1) < (N - 1) // 2, 1, 2)
    q = np.where(p["species"] == 1, 1.0, -1.0)
    q[0] = -7.0
    X = x.astype(np.longdouble)
    dx = X[:, None, :] - X[None, :, :]
    r2 = (dx ** 2).sum(-1) + d["soft"] ** 2
    np.fill_diagonal(r2, np.inf)
    ke = 1.6021766e-19 / (4 * 3.14159265358979 * 8.85419e-12)
    t = ke * q[None, :, None] * dx / r2[:, :, None] ** 1.5
    E, mag = t.sum(1), np.sqrt((t ** 2).sum(2)).sum(1)
    idx = np.resize(np.arange(N, dtype=np.uint32), 148 * 128)
    pts = np.resize(np.stack([big[a] for a in "xyz"], 1), (148 * 64, 3))
    with Run(run_config(SMALL, theta=1e-2), form="plain") as a, Run(run_config(d, dipoles=True), form="plain") as b:
        a.upload(big)
        a.build_tree()
        b.upload(p, dict(q=-7, pos=tuple(x[0])))
        b.build_tree()
        a.phi_at(pts)
        F = b.field_at(idx, x[idx])
        assert np.isfinite(F).all()
        # each of fewer than 70 terms within a few roundings, and as many in the sum
        assert (np.sqrt(((F - E[idx]) ** 2).sum(1)) <= 100 * 2.0 ** -53 * mag[idx]).all()


@pytest.mark.parametrize("N", [500, 8193, 30001])
def test_runs_from_their_start(N):
    """Ordinary runs of the plain form with dipoles: every particle stays a
    number, and the fields are the oracle's."""
    d = dict(SMALL, N=N)
    o = oracle_snapshot(d, seed=N, dipoles=True)
    o.set_grain(q=-90)
    p = o.particles()
    with Run(run_config(d, dipoles=True), form="plain", seed=2, chi_cap=True) as r:
        r.upload(p, dict(q=-90, pos=(p["x"][0], p["y"][0], p["z"][0])))
        r.build_tree()
        idx = np.arange(N, dtype=np.uint32)
        xyz = np.stack([p[a] for a in "xyz"], 1)
        F = r.field_at(idx, xyz)
        assert r.step(6)["status"] == 0
        q, _ = r.download()
    assert np.isfinite(F).all()
    assert all(np.isfinite(q[k]).all() for k in ("x", "y", "z", "vx", "vy", "vz"))
    o.build_tree()
    hi, lo = o.field_many(idx, xyz)
    ref = (np.asarray(hi, np.longdouble) + lo).astype(np.float64)
    # hundreds of terms of FP64 rounding each against sums whose parts cancel
    err = np.abs(F - ref).max(1) / np.linalg.norm(ref, axis=1)
    assert err.max() < 1e-11, err.max()
