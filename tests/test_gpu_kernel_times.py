"""Times of kernels against one another on one system (dp_time_kernel)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _liquid(counts, precision, r_cut=3.0, skin=0.3):
    from dompap_gb300 import Simulation

    dim = len(counts)
    rng = np.random.default_rng(dim)
    spacing = 0.8 ** (-1 / dim)
    box = np.array(counts) * spacing
    pos = np.stack(np.meshgrid(*[np.arange(c) for c in counts], indexing="ij"), axis=-1).reshape(-1, dim) * spacing
    pos = pos + rng.normal(0.0, 0.05, size=pos.shape)
    pos -= np.floor(pos / box) * box
    np.random.seed(4)
    sim = Simulation(positions=pos, velocities=rng.normal(size=pos.shape), box_vectors=box, masses=np.ones(len(pos)),
                     particle_types=np.zeros(len(pos), dtype=np.int32), neighbor_list_skin=skin,
                     max_number_of_neighbors=256, precision=precision)
    sim.set_pair_potential("4*(r**-12-r**-6)", r_cut)
    sim.set_neighbor_list(skin=skin, max_number_of_neighbors=256, method_str="cell list")
    sim.set_integrator(time_step=0.004, target_temperature=1.0, temperature_damping_time=0.1)
    return sim


def _time(sim, kernel, reps=10):
    from dompap_gb300 import _lib

    ms = _lib.ctypes.c_float(0.0)
    best = np.inf
    for _ in range(3):
        _lib.check(_lib.load().dp_time_kernel(sim._h, kernel, reps, _lib.ctypes.byref(ms)))
        best = min(best, ms.value)
    return best


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_forces_cost_less_than_a_step(precision):
    """The fused step walks the same lists and integrates besides."""
    from dompap_gb300 import _lib

    sim = _liquid((1000, 1000), precision)
    sim.run(5)
    assert _time(sim, _lib.DP_KERNEL_FORCES) <= _time(sim, _lib.DP_KERNEL_STEP)


@pytest.mark.parametrize("cells", [(5, 5, 5), (8, 8, 8)])
def test_small_system_step_is_the_one_that_runs(cells):
    """Up to 8,192 particles a run's steps rebuild their own lists; a step without a
    rebuild costs less than the mean step of a run, and more than a third of it."""
    from dompap_gb300 import Simulation, _lib
    from dompap_gb300.positions import FCC

    np.random.seed(1)
    sim = Simulation()
    sim.set_positions(unit_cell_coordinates=FCC, cells=cells, lattice_constants=(1.0, 1.0, 1.0))
    sim.set_masses(masses=1.0)
    sim.set_density(density=0.8442)
    sim.set_random_velocities(temperature=1.0)
    sim.set_pair_potential(pair_potential_str="4*(r**-12-r**-6)", r_cut=2.5)
    sim.set_neighbor_list(skin=0.5, max_number_of_neighbors=192)
    sim.set_integrator(time_step=0.005, target_temperature=1.0, temperature_damping_time=0.1)
    sim.run(200)
    before = np.array(sim.positions), sim._stats().steps
    step = _time(sim, _lib.DP_KERNEL_STEP, 50)
    assert np.array_equal(np.array(sim.positions), before[0]) and sim._stats().steps == before[1]
    mean = min(sim.run_timed(1000) for _ in range(3)) / 1000
    assert mean / 3 <= step <= mean
