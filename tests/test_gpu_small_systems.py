"""Systems of at most a warp per particle: the step that rebuilds its own lists
against the separate kernels, at sizes around its launch shapes, through list
overflows, far positions and either list method; sums with a warp or four
lanes per particle against the oracle's."""
import numpy as np
import pytest

from oracle import numpy_ref as ref

pytestmark = pytest.mark.gpu

LJ = "4*(r**-12-r**-6)"


def _liquid(n, seed=0, dim=3, density=0.8):
    """A jittered lattice with the first n sites occupied."""
    rng = np.random.default_rng([n, seed])
    side = int(np.ceil(n ** (1 / dim)))
    box = np.full(dim, side * density ** (-1 / dim))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * dim, indexing="ij"), axis=-1).reshape(-1, dim)[:n]
    pos = (grid + 0.5) * box / side + rng.normal(0, 0.03, size=(n, dim))
    return pos - np.floor(pos / box) * box, rng.normal(size=(n, dim)), box


def _sim(pos, vel, box, precision, skin=0.3, capacity=200, method="double loop"):
    from dompap_gb300 import Simulation

    np.random.seed(5)
    sim = Simulation(positions=pos, velocities=vel, box_vectors=box, masses=np.ones(len(pos)),
                     particle_types=np.zeros(len(pos), dtype=np.int32), neighbor_list_skin=skin,
                     max_number_of_neighbors=capacity, precision=precision)
    sim.set_pair_potential(LJ, 2.0)
    sim.set_neighbor_list(skin=skin, max_number_of_neighbors=capacity, method_str=method)
    sim.set_integrator(time_step=0.004, target_temperature=1.1, temperature_damping_time=0.1)
    return sim


def _state(sim):
    return (np.array(sim.positions), np.array(sim.velocities), np.array(sim.betas), np.array(sim.image_positions),
            sim.number_of_neighbor_list_updates)


@pytest.mark.parametrize("n", [151, 152, 304, 500, 1217, 3071, 3072, 8192, 8193])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("method", ["double loop", "cell list"])
def test_steps_match_separate_kernels(monkeypatch, n, precision, method):
    pos, vel, box = _liquid(n)
    out = []
    for fused in ("1", "0"):
        monkeypatch.setenv("DOMPAP_FUSED_STEP", fused)
        sim = _sim(pos, vel, box, precision, method=method)
        sim.run(41)
        sim.run_leap_frog(20)
        sim.run(1)
        out.append(_state(sim))
    a, b = out
    # sums in another order, amplified over 62 steps of a liquid
    tol = 1e-9 if precision == "fp64" else 2e-5
    assert np.max(np.abs(a[0] - b[0])) <= tol and np.max(np.abs(a[1] - b[1])) <= 20 * tol
    assert np.max(np.abs(a[2] - b[2])) <= 20 * tol and np.array_equal(a[3], b[3])
    assert a[4] == b[4] >= 3


@pytest.mark.parametrize("dim", [2, 3, 4])
def test_overflow_is_replayed_and_lists_stay_exact(dim):
    """A capacity far too small: the run grows it and repeats the steps; the
    list a run leaves behind is the double loop's at its reference positions."""
    pos, vel, box = _liquid(700, dim=dim)
    wide, narrow = _sim(pos, vel, box, "fp64"), _sim(pos, vel, box, "fp64", capacity=3)
    for sim in (wide, narrow):
        sim.run(60)
    a, b = _state(wide), _state(narrow)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and np.array_equal(a[3], b[3])
    narrow.max_number_of_neighbors = 200
    want, _ = ref.neighbor_list_double_loop(np.array(narrow.positions_neighbour_list), box, 2.3, 200)
    assert np.array_equal(narrow.neighbor_list, want)


def test_far_positions_take_the_reference_rules(monkeypatch):
    """Positions outside the box at the first step (wrapped by it), so that the
    list's reference positions are unwrapped until the next rebuild."""
    pos, vel, box = _liquid(400)
    pos = pos + box * np.random.default_rng(2).integers(-1, 2, size=pos.shape)
    out = []
    for fused in ("1", "0"):
        monkeypatch.setenv("DOMPAP_FUSED_STEP", fused)
        sim = _sim(pos, vel, box, "fp64")
        sim.run(30)
        out.append(_state(sim))
    a, b = out
    assert np.max(np.abs(a[0] - b[0])) <= 1e-9 and np.array_equal(a[3], b[3]) and a[4] == b[4]


def test_launch_shapes_set_by_hand(monkeypatch):
    """Lanes 1 and 4 leave the own-list step (conditional rebuild nodes again)."""
    pos, vel, box = _liquid(900)
    out = []
    for lanes in (0, 1, 4, 32):
        sim = _sim(pos, vel, box, "fp64")
        sim.set_step_launch(lanes, 0)
        sim.run(50)
        out.append(_state(sim))
    for b in out[1:]:
        assert np.max(np.abs(out[0][0] - b[0])) <= 1e-9 and out[0][4] == b[4]


@pytest.mark.parametrize("n", [33, 257, 1000, 8192, 8200])
def test_sums_match_the_oracle(n):
    pos, vel, box = _liquid(n)
    sim = _sim(pos, vel, box, "fp64")
    u, f, c = ref.make_pair_potential(LJ, 2.0)
    nl = sim.neighbor_list
    want = ref.forces_neighbor_list(pos, box, f, nl)
    got = sim.get_forces()
    assert np.sqrt(np.mean((got - want) ** 2) / np.mean(want ** 2)) <= 1e-10
    scale = ref.pair_terms_abs_sum(pos, box, u, nl)
    assert abs(sim.get_potential_energy() - ref.energy_neighbor_list(pos, box, u, nl)) <= 1e-10 * scale
    d = pos[:, None, :] - pos[nl.clip(min=0)]
    d -= box * np.round(d / box)
    r = np.where(nl >= 0, np.linalg.norm(d, axis=2), 1e9)
    inside = r <= 2.0
    fr = np.where(inside, 48 * r ** -13.0 - 24 * r ** -7.0, 0.0)
    cr = np.where(inside, 624 * r ** -14.0 - 168 * r ** -8.0, 0.0)
    assert abs(sim.get_virial() - np.sum(fr * r) / 6) <= 1e-10 * np.sum(np.abs(fr * r))
    lap = np.sum(cr - 2 * fr / r, axis=1)
    assert np.max(np.abs(sim.get_laplacian() - lap)) <= 1e-10 * np.max(np.abs(cr).sum(axis=1))


@pytest.mark.parametrize("n", [700, 9000])
def test_the_list_is_checked_again_after_every_change(n):
    """Calls that read a system skip the list check only while nothing has
    moved: after each kind of change the forces are those of a new system."""
    pos, vel, box = _liquid(n)
    sim = _sim(pos, vel, box, "fp64", method="cell list")
    rng = np.random.default_rng(4)

    def shift():
        p = np.array(sim.positions)
        p += rng.uniform(0, 1, size=3) * box + rng.normal(0, 0.05, size=p.shape)
        sim.positions = p - np.floor(p / np.array(sim.box_vectors)) * np.array(sim.box_vectors)

    def in_place():
        sim.positions[: n // 2, 0] += 0.4
        sim.wrap_into_box()

    changes = [shift, in_place, lambda: sim.run(40), lambda: sim.run_leap_frog(9), lambda: sim.scale_box(1.01), shift,
               lambda: sim.set_neighbor_list(skin=0.5), lambda: sim.step(), lambda: sim.scale_box(0.995)]
    for change in changes:
        sim.get_forces(), sim.get_potential_energy()
        change()
        other = _sim(np.array(sim.positions), vel, np.array(sim.box_vectors), "fp64", skin=float(sim.neighbor_list_skin),
                     method="cell list")
        f, g = sim.get_forces(), other.get_forces()
        # the same pairs, summed in the order of another list
        assert np.max(np.abs(f - g)) <= 1e-10 * np.max(np.abs(g))
        assert abs(sim.get_virial() - other.get_virial()) <= 1e-9 * np.sum(np.abs(g))
        assert np.allclose(sim.get_laplacian(), other.get_laplacian(), rtol=1e-9, atol=1e-9 * np.max(np.abs(g)))
