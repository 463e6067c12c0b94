"""Grouped steps (one rebuild node per group in a loop on the device) against
the graphs with gated rebuild kernels, bit for bit: step counts around the
group's length, rebuilds inside groups, either buffer set current at the
start, masses and types that move with their particles, overflow replays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(monkeypatch, conditional, dim, precision, mixture, capacity):
    from dompap_gb300 import Simulation

    monkeypatch.setenv("DOMPAP_CONDITIONAL_GRAPHS", "1" if conditional else "0")
    side = {2: 95, 3: 21, 4: 10}[dim]
    rng = np.random.default_rng(dim)
    box = np.full(dim, float(side))
    pos = np.stack(np.meshgrid(*[np.arange(side)] * dim, indexing="ij"), axis=-1).reshape(-1, dim) + 0.5
    pos = pos + rng.normal(0.0, 0.05, size=pos.shape)
    pos -= np.floor(pos / box) * box
    n = len(pos)
    types = (rng.random(n) < 0.5).astype(np.int32) if mixture else np.zeros(n, dtype=np.int32)
    np.random.seed(9)
    sim = Simulation(positions=pos, velocities=rng.normal(0.0, 1.0, size=pos.shape), box_vectors=box,
                     masses=np.where(types == 0, 1.0, 2.0), particle_types=types, neighbor_list_skin=0.3,
                     max_number_of_neighbors=capacity, precision=precision)
    if dim == 4:
        sim.set_pair_potential("(1-r/1.4)**2", 1.4)
    else:
        sim.set_pair_potential("4*(r**-12-r**-6)", 2.5)
    if mixture:
        sim.set_pair_potential_parameters(sigma=np.array([[1.0, 0.9], [0.9, 0.8]]), epsilon=np.ones((2, 2)))
    sim.set_neighbor_list(skin=0.3, max_number_of_neighbors=capacity, method_str="cell list")
    sim.set_integrator(time_step=0.004, target_temperature=1.0, temperature_damping_time=0.1)
    return sim


def _result(sim):
    return [np.array(sim.positions), np.array(sim.velocities), np.array(sim.betas), np.array(sim.image_positions),
            np.array(sim.number_of_neighbor_list_updates), np.array(sim.number_of_steps)]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dim,mixture", [(2, False), (3, False), (3, True), (4, False)])
def test_same_trajectory_as_gated_rebuilds(monkeypatch, dim, mixture, precision):
    out = []
    for conditional in (True, False):
        sim = _system(monkeypatch, conditional, dim, precision, mixture, 128)
        for steps in (1, 11, 12, 13, 0, 7, 64):
            sim.run(steps)
        sim.run_leap_frog(25)
        for _ in range(3):
            sim.step()
        assert sim._stats().conditional_graphs == int(conditional)
        out.append(_result(sim))
    assert out[0][4] >= 4
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_overflow_inside_a_group_is_replayed(monkeypatch):
    a, b = (_system(monkeypatch, True, 3, "fp32", False, c) for c in (128, 40))
    for sim in (a, b):
        sim.run(77)
    for x, y in zip(_result(a)[:4], _result(b)[:4]):
        assert np.array_equal(x, y)


def test_launch_count(monkeypatch):
    """Without a rebuild, a run is the steps and a few one-thread kernels per group."""
    from dompap_gb300 import _lib

    sim = _system(monkeypatch, True, 3, "fp32", False, 128)
    sim.set_integrator(time_step=1e-5)
    before = sim._stats().rebuilds
    sim.run(24)
    assert sim._stats().rebuilds == before
    assert int(_lib.load().dp_kernel_launches(sim._h)) == 24 + 2 * 2 + 1
