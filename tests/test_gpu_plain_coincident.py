"""A target of the plain walk at another particle's position: the status says
so (pot.c:1800-1802), that target alone is given no field, and the others'
fields are what they were."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from pot_b200.gpu import PARTICLE_DTYPE, PotError, Run
from tests.common import SMALL, run_config

pytestmark = pytest.mark.gpu

E_COINCIDENT = -5


def _plasma(N, **over):
    d = dict(SMALL, N=N, dt=2.0 ** -48, **over)
    R = d["r"] * d["mpp"]
    rng = np.random.default_rng(N)
    x = R + rng.uniform(-0.4 * R, 0.4 * R, size=(N, 3))
    x[0] = R
    p = np.zeros(N, PARTICLE_DTYPE)
    for k, a in enumerate("xyz"):
        p[a] = x[:, k]
    p["species"][1:] = np.where(np.arange(N - 1) < (N - 1) // 2, 1, 2)
    return d, p, x


@pytest.mark.parametrize("soft", [0.0, SMALL["soft"]], ids=["unsoftened", "softened"])
@pytest.mark.parametrize("over", [{}, dict(dipoles=True), dict(A=2.0)], ids=["sphere", "dipoles", "spheroid"])
@pytest.mark.parametrize("nq", [3, 8193, 32771])  # 2, 4 and 8 targets a warp
def test_query(nq, over, soft):
    N = 700
    d, p, x = _plasma(N, soft=soft, **over)
    idx = np.resize(np.arange(1, N, dtype=np.uint32), nq)
    pts = x[idx].copy()
    with Run(run_config(d), form="plain") as r:
        r.upload(p, dict(q=-5, pos=tuple(x[0])))
        r.build_tree()
        want = r.field_at(idx, pts)
        pts[1] = x[300]  # particle 2's field where particle 300 is
        got = np.full_like(pts, 1.0)
        rc = r.lib.pot_gpu_field_at(r.h, nq, idx.ctypes.data_as(C.c_void_p), pts.ctypes.data_as(C.c_void_p),
                                    got.ctypes.data_as(C.c_void_p))
    assert rc == E_COINCIDENT
    assert (got[1] == 0.0).all(), got[1]
    want[1] = 0.0
    # a list's entries can be shared out otherwise than before: the sums' rounding
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("soft", [0.0, SMALL["soft"]], ids=["unsoftened", "softened"])
def test_push(soft):
    """An electron whose half drift ends on another particle goes on without a
    field: no magnetic field, so in a straight line."""
    N = 700
    d, p, x = _plasma(N, soft=soft)
    i, j = 500, 600
    p["vx"][i] = 2.0 ** 19  # half a step: 2^-30 m
    p["x"][j] = p["x"][i] + 2.0 ** -30
    p["y"][j], p["z"][j] = p["y"][i], p["z"][i]
    out = p.copy()
    with Run(run_config(d), form="plain") as r:
        with pytest.raises(PotError) as e:
            r.move_particles(out, dict(q=-5, pos=tuple(x[0])))
    assert e.value.status == E_COINCIDENT
    assert out["vx"][i] == 2.0 ** 19 and out["vy"][i] == 0.0 and out["vz"][i] == 0.0
    assert out["x"][i] == (p["x"][i] + 2.0 ** -30) + 2.0 ** -30
    for k in ("x", "y", "z", "vx", "vy", "vz"):
        assert np.isfinite(out[k]).all(), k
