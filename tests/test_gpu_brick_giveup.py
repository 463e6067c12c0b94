"""Float32 systems of very uneven density, with enough neighbours on average for
the brick pair kernels: where a region does not fit in shared memory the bricks
are given up, and lists, sums and steps run on lists of slots. Everything
against the float64 mode of the same system."""
import numpy as np
import pytest

from test_gpu_bricks import _lattice, _rows, _sim

pytestmark = pytest.mark.gpu


def _slab():
    """A liquid of density 0.8442 filling 40 % of a long box, vacuum above it."""
    rng = np.random.default_rng(21)
    pos, size = _lattice((57, 57, 45), 60.0 / 57, rng, 0.05)
    box = np.array([60.0, 60.0, 120.0])
    pos = pos - np.floor(pos / box) * box
    # (regions: room for ~1,190 entries from the mean density, ~2,640 needed)
    return pos, box, 3.0, 0.3, "4*(r**-12-r**-6)"


def _droplet():
    """2-D: a dense disc of soft particles in a thinner gas."""
    rng = np.random.default_rng(22)
    g = np.stack(np.meshgrid(np.arange(120), np.arange(120), indexing="ij"), axis=-1).reshape(-1, 2)
    drop = (g - 59.5) * 0.4 + rng.normal(0.0, 0.02, size=(len(g), 2))
    drop = drop[np.hypot(drop[:, 0], drop[:, 1]) < 23.9] + 150.0
    side = 300.0
    gas, _ = _lattice((212, 212), side / 212, rng, 0.1)
    gas = gas[np.hypot(gas[:, 0] - 150.0, gas[:, 1] - 150.0) > 24.5]
    return np.concatenate([drop, gas]), np.array([side, side]), 4.4, 0.4, "(1-r/4.4)**2"


SYSTEMS = {"slab": _slab, "droplet": _droplet}


def _pair(name):
    pos, box, r_cut, skin, potential = SYSTEMS[name]()
    n, dim = pos.shape
    cutoff = r_cut + skin
    sphere = np.pi * cutoff**2 if dim == 2 else 4 / 3 * np.pi * cutoff**3
    assert n > 8192 and n / np.prod(box) * sphere >= 32.0  # the brick pair kernels are on at the start
    return pos, box, cutoff, [_sim(pos, box, r_cut, skin, p, capacity=512, potential=potential) for p in ("fp32", "fp64")]


def _terms(name, r):
    """u (shifted to 0 at the cut), f = -u' and c = u'' of the pair potential."""
    if name == "slab":
        at = lambda x: 4 * (x**-12 - x**-6)
        return at(r) - at(3.0), 48 * r**-13 - 24 * r**-7, 624 * r**-14 - 168 * r**-8
    x = 1 - r / 4.4
    return x * x, 2 / 4.4 * x, np.full_like(r, 2 / 4.4**2)


@pytest.mark.parametrize("name", SYSTEMS)
def test_lists_and_sums(name):
    pos, box, cutoff, (a, b) = _pair(name)
    n, dim = pos.shape
    rows = np.random.default_rng(5).choice(n, 120, replace=False)
    want = _rows(pos, box, cutoff, rows)
    nl = a.neighbor_list
    for i, w in zip(rows, want):
        assert np.array_equal(nl[i][nl[i] >= 0], w)
    # the launch shape is that of the kernels on lists of slots, not the bricks'
    assert a.get_step_launch() == ((4, 6) if n <= 65536 else (1, 6))
    # sums of the sizes of the pair terms: each float32 term carries a few
    # roundings (6e-8) times the steepness of the potential (~20), and the
    # additions half a rounding of a partial sum each: 5e-6 of the sizes in all
    size_f, size_l, size_u, size_w = (np.empty(len(rows)) for _ in range(4))
    for k, (i, w) in enumerate(zip(rows, want)):
        d = pos[i] - pos[w]
        r = np.sqrt(np.sum((d - box * np.round(d / box)) ** 2, axis=1))
        r = r[r <= (3.0 if name == "slab" else 4.4)]
        u, f, c = _terms(name, r)
        size_f[k] = np.sum(np.abs(f))
        size_l[k] = np.sum(np.abs(c) + (dim - 1) * np.abs(f) / r)
        size_u[k], size_w[k] = np.sum(np.abs(u)) / 2, np.sum(np.abs(f) * r) / (2 * dim)
    f, g = a.get_forces(), b.get_forces()
    assert np.all(np.abs(f - g)[rows] <= 5e-6 * size_f[:, None])
    assert np.sqrt(np.mean((f - g) ** 2)) <= 5e-6 * np.mean(size_f)
    lap, lap64 = np.ravel(a.get_laplacian()), np.ravel(b.get_laplacian())
    assert np.all(np.abs(lap - lap64)[rows] <= 5e-6 * size_l)
    # totals: n times the mean size of the sample
    assert abs(a.get_potential_energy() - b.get_potential_energy()) <= 5e-6 * n * np.mean(size_u)
    assert abs(a.get_virial() - b.get_virial()) <= 5e-6 * n * np.mean(size_w)


@pytest.mark.parametrize("name", SYSTEMS)
def test_steps_through_rebuilds(name):
    _, box, _, (a, b) = _pair(name)
    state = []
    for sim in (a, b):
        sim.set_integrator(time_step=0.002, target_temperature=1.0, temperature_damping_time=0.1)
        before = sim.number_of_neighbor_list_updates
        sim.run_leap_frog(60)
        assert sim.number_of_neighbor_list_updates - before >= 2
        x = np.array(sim.positions) + box * np.array(sim.image_positions)
        state.append((x, np.array(sim.velocities)))
    # float32 forces: 6e-8 of ~10 forces up to ~300 a step, over 60 steps of 0.002,
    # amplified by collisions
    assert np.max(np.abs(state[0][0] - state[1][0])) <= 1e-4
    assert np.max(np.abs(state[0][1] - state[1][1])) <= 2e-3
