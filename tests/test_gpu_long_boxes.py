"""Float64-parity forces in boxes much longer than the cutoff: the fixed-point
displacement of a pair keeps its ~48 leading bits whatever the box."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CUT = 2.5


def _force_error(box, potential, power):
    """RMS relative error of the force within isolated pairs, against extended
    precision on the displacements of the same 64-bit fixed-point positions
    (X = x 2^64 / L rounded as float64 has it: in a box of 1,000 that rounding is
    of the size of the positions' own, and ten times this error)."""
    from dompap_gb300 import Simulation

    box = np.array(box, dtype=np.float64)
    dim = len(box)
    rng = np.random.default_rng(17)
    pairs = 1200
    # pairs more than a cutoff apart from one another: on a grid over the box
    per = np.maximum(1, np.floor(box / 8.0)).astype(int)
    while np.prod(per) > 4 * pairs:
        per[np.argmax(per)] = max(1, per[np.argmax(per)] // 2)
    cells = np.stack(np.meshgrid(*[np.arange(p) for p in per], indexing="ij"), axis=-1).reshape(-1, dim)
    cells = cells[rng.permutation(len(cells))[:pairs]]
    at = (cells + rng.uniform(0.35, 0.65, size=cells.shape)) * (box / per)
    to = rng.normal(size=at.shape)
    to *= (rng.uniform(0.9, 2.3, size=len(at)) / np.sqrt(np.sum(to * to, axis=1)))[:, None]
    pos = np.concatenate([at, at + to])
    pos -= np.floor(pos / box) * box
    n = len(pos)
    assert 1000 <= n <= 8192
    np.random.seed(1)
    sim = Simulation(positions=pos, velocities=np.zeros_like(pos), box_vectors=box, masses=np.ones(n),
                     particle_types=np.zeros(n, dtype=np.int32))
    sim.set_pair_potential(potential, CUT)
    sim.set_neighbor_list(skin=0.2, max_number_of_neighbors=32)
    f = sim.get_forces().astype(np.longdouble)
    fixed = np.vectorize(int, otypes=[object])(np.floor(pos * (2.0**64 / box)))
    v = (fixed[: len(at)] - fixed[len(at):] + 2**63) % 2**64 - 2**63
    d = v.astype(np.int64).astype(np.longdouble) * (box.astype(np.longdouble) / np.longdouble(2) ** 64)
    r = np.sqrt(np.sum(d * d, axis=1))
    want = (power * r ** (-power - 2))[:, None] * d
    error = np.concatenate([f[: len(at)] - want, f[len(at):] + want])
    size = np.concatenate([power * r ** (-power - 1)] * 2)
    return float(np.sqrt(np.mean(np.sum(error * error, axis=1) / size**2)))


@pytest.mark.parametrize("potential,power", [("r**-12", 12), ("r**-9", 9)])  # without and with a square root
@pytest.mark.parametrize("shape", ["square", "long"])
def test_no_worse_than_in_a_short_box(shape, potential, power):
    if shape == "square":
        boxes, short = [(1000.0,) * 2, (3239.0,) * 2, (10123.0,) * 2], (300.0, 300.0)
    else:
        boxes, short = [(30.0, 30.0, 3000.0), (30.0, 30.0, 10123.0)], (90.0, 90.0, 90.0)
    base = _force_error(short, potential, power)
    # a dozen products and a reciprocal of ~2^-47 each, as a worst case
    assert base <= 16 * 2.0**-47
    for box in boxes:
        # the same arithmetic on a displacement of ~48 bits; the positions' own 64-bit
        # fixed point adds 2^-64 of the box, a power + 2 times steeper at r >= 0.9
        grid = (power + 2) * 2.0**-64 * max(box) / 0.9
        assert _force_error(box, potential, power) <= 1.25 * base + grid
