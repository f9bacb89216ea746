"""The plain walk where overflow buckets meet a list that is already long:
clusters of 40 particles inside one cell of the deepest level (2 R / 2^21)
among thousands of single ones, in field queries, a push and the potential
energies, against direct sums."""
from __future__ import annotations

import numpy as np
import pytest

from pot_b200.gpu import PARTICLE_DTYPE, Run
from tests.common import SMALL, run_config

pytestmark = pytest.mark.gpu

KE = 1.6021766e-19 / (4 * 3.14159265358979 * 8.85419e-12)


def _clustered(seed, clusters, n=2001, size=40):
    # an opening angle at which every cell opens: the deepest cell is 2 R / 2^20 wide
    d = dict(SMALL, N=n, theta=1e-7)
    R = d["r"] * d["mpp"]
    rng = np.random.default_rng(seed)
    x = R + rng.uniform(-0.5 * R, 0.5 * R, size=(n, 3))
    x[0] = R
    for c in range(clusters):
        a = 10 + (n // clusters - 5) * c
        x[a:a + size] = x[a] + rng.uniform(0.0, 1e-9 * R, size=(size, 3))
    p = np.zeros(n, PARTICLE_DTYPE)
    for k, a in enumerate("xyz"):
        p[a] = x[:, k]
    p["species"][1:] = np.where(np.arange(n - 1) < (n - 1) // 2, 1, 2)
    q = np.where(p["species"] == 1, 1.0, -1.0)
    q[0] = -7.0
    return d, p, x, q


def _direct(d, x, q):
    """(field, sum of the terms' magnitudes, potential, the same for it) of
    every particle from all others, softened pairs, in long double."""
    X, Q = x.astype(np.longdouble), q.astype(np.longdouble)
    E, mag, phi, pmag = (np.zeros(s, np.longdouble) for s in (x.shape, len(x), len(x), len(x)))
    for i in range(len(x)):
        dx = X[i] - X
        r2 = (dx ** 2).sum(1) + np.longdouble(d["soft"]) ** 2
        w = KE * Q / r2 ** 1.5
        w[i] = 0.0
        t = w[:, None] * dx
        E[i] = t.sum(0)
        mag[i] = np.sqrt((t ** 2).sum(1)).sum()
        v = KE * Q / np.sqrt(r2)
        v[i] = 0.0
        phi[i], pmag[i] = v.sum(), np.abs(v).sum()
    return E, mag, phi, pmag


def _run(d, p):
    r = Run(run_config(d), form="plain")
    r.upload(p, dict(q=-7, pos=(p["x"][0], p["y"][0], p["z"][0])))
    return r


# A term's error: a few roundings of its own plus those of the sum, at most
# N / 2^53 = 2.2e-13 of the terms' magnitudes for 2,001 terms added in any order.
TOL = 2.5e-13


@pytest.mark.parametrize("clusters", [10, 20])
@pytest.mark.parametrize("nq", [2001, 40001])  # two and eight targets a warp
def test_field_query(clusters, nq):
    d, p, x, q = _clustered(clusters, clusters)
    E, mag, _, _ = _direct(d, x, q)
    idx = np.resize(np.arange(len(x), dtype=np.uint32), nq)
    with _run(d, p) as r:
        r.build_tree()
        F = r.field_at(idx, x[idx])
    err = np.sqrt(((F - E[idx]) ** 2).sum(1))
    assert (err <= TOL * mag[idx]).all(), float((err / mag[idx]).max())


@pytest.mark.parametrize("clusters", [10, 20])
def test_step_with_energies(clusters):
    """A step from rest with no magnetic field: each electron's velocity change
    is its field's, and the energies are the species' sums of q phi."""
    d, p, x, q = _clustered(3 + clusters, clusters)
    d = dict(d, a=1e-12)
    E, mag, phi, pmag = _direct(d, x, q)
    with _run(d, p) as r:
        st = r.step(1, epe=True)
        out, _ = r.download()
    e = np.flatnonzero(p["species"] == 2)
    v = np.stack([out[a] for a in ("vx", "vy", "vz")], 1)[e]
    qom_dt = -1.6021766e-19 / 9.109383e-31 * d["dt"]
    err = np.sqrt(((v / qom_dt - E[e]) ** 2).sum(1))
    assert (err <= 2 * TOL * mag[e]).all(), float((err / mag[e]).max())
    for sp in (1, 2):
        m = p["species"] == sp
        want = float((1.6021766e-19 * q[m] * phi[m]).sum())
        assert abs(st["epe"][sp] - want) <= 2 * TOL * float((1.6021766e-19 * pmag[m]).sum())
