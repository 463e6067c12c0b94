"""Lists built brick by brick on the tensor cores, and the float32 pair kernels
that run on the bricks: the pair set against a float64 all-pairs list over
dimensions, box shapes, densities and particle numbers that leave bricks
partly filled, empty or overfull; forces, energy, virial and Laplacian
against the float64 mode; steps against the kernels on lists of slots."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LJ = "4*(r**-12-r**-6)"


def _sim(pos, box, r_cut, skin, precision="fp32", method="cell list", capacity=256, types=None, potential=LJ):
    from dompap_gb300 import Simulation

    n = len(pos)
    np.random.seed(11)
    sim = Simulation(positions=pos, velocities=np.random.default_rng(1).normal(size=pos.shape), box_vectors=box,
                     masses=np.ones(n), particle_types=np.zeros(n, dtype=np.int32) if types is None else types,
                     neighbor_list_skin=skin, max_number_of_neighbors=capacity, precision=precision)
    sim.set_pair_potential(potential, r_cut)
    if types is not None:
        sim.set_pair_potential_parameters(sigma=np.array([[1.0, 0.9], [0.9, 0.8]]), epsilon=np.array([[1.0, 1.5], [1.5, 0.5]]))
    sim.set_neighbor_list(skin=skin, max_number_of_neighbors=capacity, method_str=method)
    return sim


def _lattice(counts, spacing, rng, jitter):
    grid = np.stack(np.meshgrid(*[np.arange(c) for c in counts], indexing="ij"), axis=-1).reshape(-1, len(counts))
    box = np.array(counts, dtype=np.float64) * spacing
    pos = (grid + 0.5) * spacing + rng.normal(0.0, jitter, size=grid.shape)
    return pos - np.floor(pos / box) * box, box


def _rows(pos, box, cutoff, rows):
    """Partners of some particles by the list's float64 rule."""
    out = []
    for i in rows:
        d = pos[i] - pos
        d = np.where(d > box / 2, d - box, np.where(d < -box / 2, d + box, d))
        q = d[:, 0] * d[:, 0]
        for k in range(1, pos.shape[1]):
            q = q + d[:, k] * d[:, k]
        m = np.nonzero(np.sqrt(q) < cutoff)[0]
        out.append(m[m != i])
    return out


# (particles per axis, spacing, r_cut, skin): 3 to 11 cells per axis, odd numbers,
# long and flat boxes, crowded cells, 2-D and 4-D
SHAPES = [((23, 22, 21), 1.05, 2.5, 0.4), ((60, 14, 13), 1.0, 2.5, 0.5), ((9, 40, 40), 1.05, 2.5, 0.3),
          ((33, 31, 30), 0.6, 2.0, 0.2), ((120, 110), 1.0, 4.0, 0.5), ((12, 12, 11, 10), 1.0, 1.9, 0.2),
          ((22, 22, 22), 1.0, 6.9, 0.1)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s[0])))
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_pair_set_is_exact(shape, precision):
    counts, spacing, r_cut, skin = shape
    rng = np.random.default_rng(sum(counts))
    pos, box = _lattice(counts, spacing, rng, 0.15 * spacing)
    # some pairs exactly at the cutoff, and some a rounding away from it
    pos[1] = pos[0] + np.eye(len(counts))[0] * (r_cut + skin)
    pos[3] = pos[2] + np.eye(len(counts))[1] * np.nextafter(r_cut + skin, 0.0)
    pos -= np.floor(pos / box) * box
    sim = _sim(pos, box, r_cut, skin, precision, capacity=64, potential="(1-r/10)**2")
    n = len(pos)
    rows = np.concatenate([[0, 1, 2, 3], rng.choice(n, 150, replace=False)])
    want = _rows(pos, box, r_cut + skin, rows)
    sim.max_number_of_neighbors = max(len(w) for w in want) + 2
    nl = sim.neighbor_list
    for i, w in zip(rows, want):
        assert np.array_equal(nl[i][nl[i] >= 0], w)
    # the export left the lists usable
    assert np.all(np.isfinite(sim.get_forces()))


def test_uneven_density_grows_or_gives_up_the_regions():
    """A dense drop in a thin gas: its regions exceed the capacity that the mean
    density suggests by a lot."""
    rng = np.random.default_rng(8)
    drop, _ = _lattice((30, 30, 30), 0.5, rng, 0.02)
    gas = rng.uniform(0.0, 40.0, size=(3000, 3))
    gas = gas[np.any(np.abs(gas - 27.5) > 9.0, axis=1)]
    pos, box = np.concatenate([drop + 20.0, gas]), np.array([40.0, 40.0, 40.0])
    sim = _sim(pos, box, 2.0, 0.3, capacity=64, potential="(1-r/10)**2")
    rows = np.concatenate([rng.choice(27000, 60, replace=False), np.arange(27000, 27040)])
    want = _rows(pos, box, 2.3, rows)
    sim.max_number_of_neighbors = max(len(w) for w in want) + 2
    nl = sim.neighbor_list
    for i, w in zip(rows, want):
        assert np.array_equal(nl[i][nl[i] >= 0], w)
    sim.set_integrator(time_step=1e-4)
    sim.run_leap_frog(3)
    assert np.all(np.isfinite(sim.positions))


@pytest.mark.parametrize("shape", [s for s in SHAPES if len(s[0]) < 4 and np.prod(s[0]) > 8192],
                         ids=lambda s: "x".join(map(str, s[0])))
@pytest.mark.parametrize("mixture", [False, True])
def test_pair_sums_match_float64(shape, mixture):
    counts, spacing, r_cut, skin = shape
    rng = np.random.default_rng(3)
    pos, box = _lattice(counts, spacing, rng, 0.04 * spacing)
    pot = f"4*((r/{spacing!r})**-12-(r/{spacing!r})**-6)"
    types = (np.arange(len(pos)) % 2).astype(np.int32) if mixture else None
    a = _sim(pos, box, r_cut, skin, "fp32", types=types, capacity=64, potential=pot)
    b = _sim(pos, box, r_cut, skin, "fp64", types=types, capacity=64, potential=pot)
    f, g = a.get_forces(), b.get_forces()
    # float32 pair terms: a few roundings (6e-8) of terms up to ~20 times the sum
    assert np.sqrt(np.mean((f - g) ** 2) / np.mean(g ** 2)) <= 5e-6
    lap, lap64 = a.get_laplacian(), b.get_laplacian()
    assert np.sqrt(np.mean((lap - lap64) ** 2) / np.mean(lap64 ** 2)) <= 5e-6
    assert abs(a.get_potential_energy() - b.get_potential_energy()) <= 5e-6 * abs(b.get_potential_energy())
    assert abs(a.get_virial() - b.get_virial()) <= 2e-5 * np.sum(np.abs(f)) * spacing / 3


@pytest.mark.parametrize("lanes", [0, 1, 4, 32])
@pytest.mark.parametrize("nve", [False, True])
def test_steps_match_the_other_kernels(monkeypatch, lanes, nve):
    """12,000 particles, through several rebuilds, with every launch shape,
    against the separate force and integrator kernels on the same lists and
    against one warp per particle on lists of slots (lanes = 32)."""
    def trajectory(shape, fused="1"):
        monkeypatch.setenv("DOMPAP_FUSED_STEP", fused)
        rng = np.random.default_rng(6)
        pos, box = _lattice((25, 24, 20), 1.06, rng, 0.05)
        sim = _sim(pos, box, 2.5, 0.3)
        sim.set_integrator(time_step=0.004, target_temperature=1.0, temperature_damping_time=0.1)
        sim.set_step_launch(shape, 0)
        (sim.run_leap_frog if nve else sim.run)(60)
        return sim._stats().rebuilds, np.array(sim.positions), np.array(sim.velocities), np.array(sim.image_positions)

    a, b = trajectory(lanes), trajectory(32)
    c = trajectory(lanes, "0")
    assert a[0] >= 3
    for other in (b, c):
        # float32 sums in another order, 6e-8 of forces up to ~300, over 60 steps
        assert np.max(np.abs(a[1] - other[1])) <= 2e-5
        assert np.max(np.abs(a[2] - other[2])) <= 5e-4
