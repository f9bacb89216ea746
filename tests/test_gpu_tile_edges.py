"""Particle counts around the tiles of the tree build (radix pass, cell
numbering, due list) and around the sort's change of tile size: the tree
against the oracle's, and a step captured on several streams against the same
kernels run one after another."""
from __future__ import annotations

import numpy as np
import pytest

from common import SMALL, by_cell, canonical_dump, oracle_snapshot, run_config
from pot_b200.gpu import Run
from test_gpu_parity import gpu_from_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1024, 1025, 2048, 2049, 2050, 4096, 4097, 99999, 100000])
def test_tree_at_tile_edges(N):
    d = dict(SMALL, N=N)
    o = oracle_snapshot(d, seed=3, mode="gpu")
    o.set_grain(q=-40)
    o.build_tree()
    od = o.tree_dump()
    with gpu_from_oracle(d, o) as r:
        assert r.build_tree() == len(od["int_level"])
        gd = r.tree_dump()
    assert canonical_dump(gd) == canonical_dump(od)
    assert by_cell(gd) == by_cell(od)


@pytest.mark.parametrize("form", ["plain", "fast"])
@pytest.mark.parametrize("N", [1025, 4096, 4097, 8193])
def test_captured_steps_equal_kernel_by_kernel(N, form):
    """timing=True launches each kernel alone on one stream; without it the
    first step of each parity does too and later ones replay a forked graph.
    The same kernels on the same data: equal bits."""
    out = []
    for timing in (True, False):
        with Run(run_config(dict(SMALL, N=N)), form=form, seed=9, chi_cap=True, timing=timing) as r:
            r.init_particles()
            st = [r.step(1) for _ in range(3)] + [r.step(4)]
            p, g = r.download()
            out.append((p.tobytes(), [{k: v for k, v in z.items() if k != "epe"} for z in st],
                        {k: np.asarray(v).tobytes() for k, v in g.items()}))
    assert out[0][1] == out[1][1]  # every statistic of every step
    assert out[0][2] == out[1][2]  # the grain
    assert out[0][0] == out[1][0]  # the particles
