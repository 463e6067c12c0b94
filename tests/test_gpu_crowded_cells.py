"""Cells of more entries than the counting sort holds in shared memory (48): the
slots of a cell come out in ascending order of their ids, whatever order the
atomics left them in, so lists and float32 sums repeat bit for bit."""
import numpy as np
import pytest

from test_gpu_bricks import _lattice, _rows, _sim

pytestmark = pytest.mark.gpu

# (particles per axis, spacing, r_cut): ~57, ~110 (4-D), ~350 and ~1,450 entries a cell
SYSTEMS = [((30, 30, 30), 0.6, 2.0), ((13, 13, 13, 13), 1.0, 2.9), ((22, 22, 22), 1.0, 6.7), ((120, 110), 1.0, 33.0)]


@pytest.mark.parametrize("system", SYSTEMS, ids=lambda s: "x".join(map(str, s[0])))
def test_lists_repeat(system):
    counts, spacing, r_cut = system
    rng = np.random.default_rng(len(counts))
    pos, box = _lattice(counts, spacing, rng, 0.1 * spacing)
    order = rng.permutation(len(pos))  # ids in no spatial order
    pos = pos[order]
    cells = np.prod(np.floor(box / (r_cut + 0.2)))
    assert len(pos) / cells > 48 and np.all(np.floor(box / (r_cut + 0.2)) >= 3)
    rows = rng.choice(len(pos), 40, replace=False)
    want = _rows(pos, box, r_cut + 0.2, rows)
    out = []
    for _ in range(2):
        sim = _sim(pos, box, r_cut, 0.2, "fp32", capacity=64, potential=f"(1-r/{r_cut})**2")
        sim.max_number_of_neighbors = max(len(w) for w in want) + 64
        nl = sim.neighbor_list
        for i, w in zip(rows, want):
            assert np.array_equal(nl[i][nl[i] >= 0], w)
        sim.set_integrator(time_step=0.01)
        sim.run_leap_frog(40)
        out.append((np.array(sim.positions), np.array(sim.velocities)))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
