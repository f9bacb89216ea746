"""The fast push by pairs of warps (runs of few groups) against the same run
stepped in a packed batch, whose walk is one warp per group: the same sums in
the same order, so the same bits, on group sizes that split the warp and with
one and two targets per lane."""
from __future__ import annotations

import numpy as np
import pytest

from pot_b200.gpu import Batch, Run
from tests.common import SMALL, STRESS, run_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", [8, 16, 32, 64])
@pytest.mark.parametrize("d,N,leaf", [(SMALL, 40, 8), (SMALL, 8193, 8), (STRESS, 4097, 16)],
                         ids=["few", "small", "stress"])
def test_pair_walk_is_the_one_warp_walk(d, N, leaf, group):
    cfg = run_config(d, N=N)
    with Run(cfg, form="fast", leaf_size=leaf, group_size=group, seed=7, chi_cap=True) as r, Batch() as b:
        r.init_particles()
        st = r.step(6)
        slot = b.admit(cfg, leaf_size=leaf, group_size=group, seed=7, chi_cap=True)
        b.step(6)
        p, g = r.download()
        q, h = b.download(slot)
        rows = b.summary()
    assert st["status"] == 0 and rows["status"][0] == 0
    for k in ("x", "y", "z", "vx", "vy", "vz", "species"):
        assert np.array_equal(p[k], q[k]), k
    assert g["q"] == h["q"] and g["chi_b"] == h["chi_b"]
