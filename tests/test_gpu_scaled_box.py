"""A box that is scaled step by step: the bricks' buffers are kept and only grow, and
lists and forces are those of a system made in that box."""
import numpy as np
import pytest

from test_gpu_bricks import _lattice, _rows, _sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_lists_and_forces_follow_the_box(precision):
    rng = np.random.default_rng(41)
    pos, box = _lattice((26, 25, 24), 1.06, rng, 0.05)
    sim = _sim(pos, box, 2.5, 0.3, precision, capacity=192)
    # fewer and more cells and bricks, and back
    for factor in (0.93, 0.94, 1.30, 1.05, 0.80, 1.02):
        sim.scale_box(factor)
        new, size = np.array(sim.positions), np.array(sim.box_vectors)
        rows = rng.choice(len(new), 30, replace=False)
        nl = sim.neighbor_list
        for i, w in zip(rows, _rows(new, size, 2.8, rows)):
            assert np.array_equal(nl[i][nl[i] >= 0], w)
        other = _sim(new, size, 2.5, 0.3, precision, capacity=192)
        f, g = sim.get_forces(), other.get_forces()
        # the same pair terms; the lists may hold them in another order (float32:
        # roundings of 6e-8, float64: of the double-float sums, 2^-45)
        assert np.sqrt(np.mean((f - g) ** 2) / np.mean(g**2)) <= (5e-6 if precision == "fp32" else 1e-12)
        sim.run_leap_frog(1)
