"""Device memory of a fast run, bytes per particle: node records are kept for
the children that exist, not for eight places of every cell.  The bounds are
what the runs took when a cell's moments were two arrays of 20 bytes a node
(leaf size 1, whose leaves had none, a tenth more)."""
import pytest

from pot_b200.gpu import RunConfig, bytes_needed

BOUND = {1: 1.1 * 794.6, 2: 1050.3, 4: 708.3, 8: 537.3, 16: 451.8, 32: 409.0, 64: 387.7}
BOUND_DIPOLES = {1: 1.1 * 1026.9, 2: 1465.1, 4: 947.1, 8: 688.1, 16: 558.6, 32: 493.8, 64: 461.4}


@pytest.mark.parametrize("n", [1000001, 1 << 24])
@pytest.mark.parametrize("dipoles", [False, True], ids=["monopoles", "dipoles"])
def test_bytes_per_particle(n, dipoles):
    cfg = RunConfig(N=n, r=1000, dt=1e-12, mpp=4e-7, soft=2e-8, Te=220, Ti=220, a=2.5e-6, settle=0.0,
                    dipoles=dipoles)
    for leaf, bound in (BOUND_DIPOLES if dipoles else BOUND).items():
        assert bytes_needed(cfg, form="fast", leaf_size=leaf) <= bound * n, leaf
