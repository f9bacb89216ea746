"""Which status a state with several faults ends with, on a step replayed as a
graph, whose branches run side by side: the one the launches' order gives."""
from __future__ import annotations

import numpy as np
import pytest

from pot_b200.gpu import PARTICLE_DTYPE, Batch, PotError, Run
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


@pytest.mark.parametrize("form,N,integrator", [("plain", 20001, 0), ("fast", 20001, 0), ("fast", 2000001, 0),
                                               ("plain", 5001, 1), ("fast", 5001, 2)])
def test_a_failed_edge_potential_stops_the_push(form, N, integrator):
    """An edge potential that is no number (the grain's position given as NaN) on
    the 20th step: the step ends with the walk's status and no particle moves."""
    d = dict(SMALL, N=N, integrator=integrator)
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
            st = e.value.stats
            assert st["n_pushed"] == 0 and st["n_reinjected"] == 0 and st["n_absorbed"] == 0 and st["dq"] == 0
            assert st["interactions"] == 0 and st["grain_q"] == -7
        # the drop-in call gives back the records as the step found them
        r.upload(p, dict(q=-7, pos=c, t_steps=18))
        r.step(1)
        out, _ = r.download()
        kept = out.copy()
        with pytest.raises(PotError) as e:
            r.move_particles(out, dict(q=-7, pos=(np.nan, c[1], c[2]), t_steps=19))
        assert e.value.status == E_WALK
        for a in ("x", "y", "z", "vx", "vy", "vz", "species"):
            assert np.array_equal(out[a][1:], kept[a][1:]), a


def test_a_failed_edge_potential_in_a_packed_batch():
    """It undoes the step of its own run only."""
    N = 6001
    d = dict(SMALL, N=N)
    p = _state(N, d["r"] * d["mpp"], 6)
    c = (p["x"][0], p["y"][0], p["z"][0])
    cfg = run_config(d)
    o = dict(leaf_size=8, seed=9, chi_cap=True)
    with Run(cfg, form="fast", **o) as r, Batch() as b:
        r.upload(p, dict(q=-7, pos=c, t_steps=18))
        r.step(2)
        good = b.admit(cfg, parts=p, grain=dict(q=-7, pos=c, t_steps=18), **o)
        bad = b.admit(cfg, parts=p, grain=dict(q=-7, pos=(np.nan, c[1], c[2]), t_steps=18), **o)
        b.step(2)
        rows = {int(w["slot"]): w for w in b.summary()}
        want, g = r.download()
        got, h = b.download(good)
    assert rows[good]["status"] == 0 and rows[bad]["status"] == E_WALK
    assert rows[bad]["t_steps"] == rows[good]["t_steps"] == 20
    for a in ("x", "y", "z", "vx", "vy", "vz", "species"):
        assert np.array_equal(want[a], got[a]), a
    assert g["q"] == h["q"] and g["chi_b"] == h["chi_b"]
