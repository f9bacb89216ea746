"""The fast push by pairs of warps meets at a named barrier of 64 threads, which
whole warps must reach converged -- also after a push in which the lanes of the
evaluating warp part (absorbed, bounced or reinjected members, members of a
group smaller than the warp)."""
import os
import re

import numpy as np
import pytest

from pot_b200.gpu import Batch, Run
from tests.common import STRESS, run_config

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pot_b200", "csrc",
                   "pot_walk_fast.cu")


def test_named_barriers_are_reached_converged():
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    at = [m.start() for m in re.finditer(r"bar\.sync", text)]
    assert at
    for a in at:
        before = text[:a].rsplit("{", 1)[-1]  # the statements of its function ahead of it
        assert before.split()[:1] == ["__syncwarp();"], before


@pytest.mark.gpu
@pytest.mark.parametrize("group", [8, 32, 64])
@pytest.mark.parametrize("over", [dict(bounce=0.7, dt=2e-13), dict(A=3.0, a=2e-7, dt=1e-13), dict(a=4e-7)],
                         ids=["wall", "spheroid", "grain"])
def test_parted_lanes_give_the_one_warp_push(over, group):
    d = dict(STRESS, **over)
    cfg = run_config(d)
    with Run(cfg, form="fast", leaf_size=8, group_size=group, seed=3, chi_cap=True) as r, Batch() as b:
        r.init_particles()
        st = r.step(4)
        slot = b.admit(cfg, leaf_size=8, group_size=group, seed=3, chi_cap=True)
        b.step(4)
        p, g = r.download()
        q, h = b.download(slot)
        rows = b.summary()
    assert st["status"] == 0 and rows["status"][0] == 0
    assert st["n_reinjected"] + st["n_bounced"] > 0
    for k in ("x", "y", "z", "vx", "vy", "vz", "species"):
        assert np.array_equal(p[k], q[k]), k
    assert g["q"] == h["q"]
